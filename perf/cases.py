"""The work that users of shearwave_b200 have it do, as cases whose time can be measured.

Every case goes through a public function of the package, with CUDA tensors in
and out (``return_device=True`` where a function has it).  Sizes and value
distributions are those of ``shearwave_b200.workloads`` and of the tests:

``solve``     ``shear_fdtd``: one simulation, projection included.  Options:
              precision, a viscosity map / number / none, velocity damping,
              several pushes, snapshots, the compensated sum.
``batch``     ``shear_fdtd_batch``: many independent simulations at once.
``project``   ``project_vector_field``: the force projection alone, by the
              conjugate gradient or by the direct solve, float32 or float64.
``static``    ``elastic_solve_static``: the static elastic solve.
``strain``    ``compute_strain_fields`` of a displacement, or
              ``compute_strain_tensor`` followed by the invariants.
``arf``       ``compute_radiation_force`` (auto gate or a slice) and
              ``compute_radiation_force_velocity`` from recorded fields.
``operators`` ``laplacian_center``, ``divergence_center``, ``gradient_center``.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import shearwave_b200 as sw

H = 0.5e-3  # grid spacing of every workload [m]


def listed():
    return [
        # an operator on a small field: what is left is latency and launches
        dict(name="operators_64", kind="operators", nx=64, ny=64, nz=64, dtype="float32"),
        # a quick small run: homogeneous medium, one centred push, snapshots
        dict(name="solve_small_64", kind="solve", nx=64, ny=64, nz=64, n_steps=500,
             precision="mixed", medium="uniform", eta="number", pushes=1, damp=0.0, stride=10,
             kahan=False),
        # the ordinary run: heterogeneous medium with a viscosity map, snapshots
        dict(name="solve_192", kind="solve", nx=192, ny=192, nz=192, n_steps=1000,
             precision="mixed", medium="inclusions", eta="map", pushes=1, damp=0.0, stride=20,
             kahan=False),
        # the large run: stiff layer over soft tissue, eight pushes one after another
        dict(name="solve_layered_384", kind="solve", nx=256, ny=256, nz=384, n_steps=600,
             precision="mixed", medium="layered", eta="map", pushes=8, damp=0.0, stride=0,
             kahan=False),
        # the reference's arithmetic in double precision, a ragged grid, damped
        dict(name="solve_fp64_147", kind="solve", nx=147, ny=146, nz=194, n_steps=300,
             precision="fp64", medium="inclusions", eta="map", pushes=1, damp=0.002, stride=0,
             kahan=False),
        # a parameter study: independent solves of varied grids and lengths
        dict(name="batch_24", kind="batch", count=24, lo=64, hi=160, hi_z=224, steps_lo=200,
             steps_hi=800, precision="mixed"),
        # the force projection to a tight tolerance, double precision
        dict(name="project_cg_192", kind="project", nx=192, ny=192, nz=192, dtype="float64",
             method="cg", tol=1e-10, iters=600, comps=1),
        # the direct projection of a three-component force on a ragged grid
        dict(name="project_direct_173", kind="project", nx=160, ny=131, nz=173, dtype="float32",
             method="spectral", tol=1e-10, iters=600, comps=3),
        # a quasistatic displacement at the reference's default tolerance
        dict(name="static_121", kind="static", nx=121, ny=121, nz=141, dtype="float32",
             field=False, tol=1e-6, iters=1500),
        # the post-pass of the ordinary run: strain tensor and all invariants
        dict(name="strain_192", kind="strain", nx=192, ny=192, nz=192, dtype="float32",
             form="fields"),
        # radiation force of a recorded pressure, the gate found from the record
        dict(name="arf_pressure_auto", kind="arf", nx=128, ny=96, nz=112, nt=300,
             dtype="float32", velocity=False, gate="auto", maps=True),
        # the vector form: pressure and three velocity records, a given gate
        dict(name="arf_velocity_gate", kind="arf", nx=80, ny=72, nz=101, nt=257,
             dtype="float32", velocity=True, gate="slice", maps=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["operators", "solve", "solve", "solve", "solve", "batch", "project",
                       "project", "static", "strain", "arf", "arf"])
    dtype = rng.choice(["float32", "float32", "float64"])
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        top = 224 if precision == "mixed" else 160
        nx, ny, nz = _log(rng, 24, top), _log(rng, 24, top), _log(rng, 24, 1.5 * top)
        room = int((8e9 if precision == "mixed" else 3e9) / (nx * ny * nz))
        n = max(2, min(_log(rng, 20, 2000), room))
        stride = rng.choice([0, 0, 5, 10])
        if stride:
            # snapshots of at most about 2 GB
            stride = max(stride, n * nx * ny * nz * 12 // 2_000_000_000 + 1)
            n = max(stride, n - n % stride)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, n_steps=n, precision=precision,
                    medium=rng.choice(["uniform", "inclusions", "inclusions", "layered"]),
                    eta=rng.choice(["none", "number", "map", "map"]),
                    pushes=rng.choice([1, 1, 1, 2, 4]), damp=rng.choice([0.0, 0.0, 0.001]),
                    stride=stride, kahan=precision == "mixed" and rng.random() < 0.1)
    if kind == "batch":
        hi = _log(rng, 48, 160)
        lo = _log(rng, 24, hi)
        hi_z = rng.randint(hi, 224)
        top = _log(rng, 100, 700)
        return dict(kind=kind, count=rng.randint(2, 20), lo=lo, hi=hi, hi_z=hi_z,
                    steps_lo=rng.randint(top // 4, top), steps_hi=top,
                    precision=rng.choice(["mixed", "mixed", "fp64"]))
    nx, ny, nz = _log(rng, 20, 192), _log(rng, 20, 192), _log(rng, 20, 224)
    if kind == "project":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype,
                    method=rng.choice(["cg", "spectral"]), tol=rng.choice([1e-5, 1e-10]),
                    iters=600, comps=rng.choice([1, 3]))
    if kind == "static":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype, field=rng.random() < 0.3,
                    tol=rng.choice([1e-5, 1e-6]), iters=1500)
    if kind == "strain":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype,
                    form=rng.choice(["fields", "invariants", "tensor"]))
    if kind == "arf":
        nx, ny, nz = _log(rng, 20, 128), _log(rng, 20, 128), _log(rng, 20, 128)
        velocity = rng.random() < 0.4
        nt = _log(rng, 40, 1500)
        most = (1.5e9 if velocity else 4e9) / (nx * ny * nz * (4 if dtype == "float32" else 8))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nt=max(16, min(nt, int(most))), dtype=dtype,
                    velocity=velocity, gate=rng.choice(["auto", "auto", "slice", "mask"]),
                    maps=rng.random() < 0.6)
    return dict(kind=kind, nx=nx, ny=ny, nz=nz, dtype=dtype)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
DEV = "cuda"


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _axes(shape):
    ax = [torch.arange(n, device=DEV, dtype=torch.float64) * H for n in shape]
    return ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]


def _push(shape, centre, sig_lat, sig_ax, dtype, amp=1e3):
    """Axial Gaussian body force [N/m^3]."""
    x, y, z = _axes(shape)
    cx, cy, cz = centre
    r2 = ((x - cx) ** 2 + (y - cy) ** 2) / (2 * sig_lat**2) + (z - cz) ** 2 / (2 * sig_ax**2)
    return (amp * torch.exp(-r2)).to(dtype)


def _smooth(shape, rng, gen):
    """Smooth field in [-1, 1]: a few plane waves of seeded directions."""
    x, y, z = _axes(shape)
    f = torch.zeros(shape, device=DEV, dtype=torch.float64)
    for _ in range(6):
        k = rng.normal(0.0, 1.0, 3) * 2 * math.pi / 8e-3
        f += torch.cos(k[0] * x + k[1] * y + k[2] * z + rng.uniform(0, 2 * math.pi))
    return f / 6


def _medium(shape, medium, eta_kind, rng, gen, dtype):
    """(rho, mu, eta) as numbers or maps."""
    if medium == "uniform":
        rho, mu = 1000.0, 2000.0 * float(rng.uniform(0.8, 1.2))
        eta = torch.full(shape, 1.0, device=DEV, dtype=torch.float64)
    elif medium == "layered":
        zc = (torch.arange(shape[2], device=DEV, dtype=torch.float64) + 0.5) * H
        slab = ((zc >= 2.5e-3) & (zc < 7.5e-3))[None, None, :]
        var = 1.0 + 0.1 * _smooth(shape, rng, gen)
        mu = (torch.where(slab, 500e3, 2e3) * var).to(dtype)
        rho = (torch.where(slab, 1900.0, 1040.0) * var).to(dtype)
        eta = torch.where(slab, 2.0, 1.0) * var
    else:
        rho = 1000.0 * (1.0 + 0.1 * (torch.rand(shape, generator=gen, device=DEV,
                                                dtype=torch.float64) - 0.5))
        rho = rho.to(dtype)
        mu = torch.full(shape, 3e3, device=DEV, dtype=torch.float64)
        eta = torch.full(shape, 1.0, device=DEV, dtype=torch.float64)
        x, y, z = _axes(shape)
        for _ in range(12):
            c = rng.uniform(0.0, 1.0, 3) * np.array(shape) * H
            r = rng.uniform(2e-3, 8e-3)
            inside = (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 < r * r
            mu = torch.where(inside, math.exp(rng.uniform(math.log(1e3), math.log(2e4))), mu)
            eta = torch.where(inside, rng.uniform(0.5, 5.0), eta)
        mu = mu.to(dtype)
    if eta_kind == "none":
        return rho, mu, 0.0
    if eta_kind == "number":
        return rho, mu, 0.5
    return rho, mu, eta.to(dtype)


def _low(v):
    return float(v.min()) if isinstance(v, torch.Tensor) else float(v)


def _high(v):
    return float(v.max()) if isinstance(v, torch.Tensor) else float(v)


def _problem(c, seed):
    """shear_fdtd's arguments for one simulation."""
    rng, gen = np.random.default_rng(seed), _gen(seed)
    shape = (c["nx"], c["ny"], c["nz"])
    fp64 = c["precision"] == "fp64"
    dtype = torch.float64 if fp64 else torch.float32
    n = c["n_steps"]
    rho, mu, eta = _medium(shape, c["medium"], c["eta"], rng, gen, dtype)
    # elastic limit, and the explicit viscous one (eta dT 12 / (rho h^2) <= 2)
    dT = min(20e-6, 0.35 * H / math.sqrt(3.0 * _high(mu) / _low(rho)))
    if _high(eta) > 0:
        dT = min(dT, 0.9 * _low(rho) * H * H / (6.0 * _high(eta)))
    size = np.array(shape) * H
    terms = []
    for k in range(c["pushes"]):
        centre = (0.25 + 0.5 * rng.uniform(0.0, 1.0, 3)) * size
        env = np.zeros(n, np.float64 if fp64 else np.float32)
        start = 0 if k == 0 else int(rng.integers(0, max(1, n // 4)))
        env[start:start + 10] = 1.0
        terms.append((_push(shape, centre, 1.5e-3, 5e-3, dtype), env))
    opts = dict(env_t=terms[0][1], eta=eta, poisson_tol=1e-10, poisson_max_iters=3 * max(shape),
                precision=c["precision"])
    if len(terms) > 1:
        opts["force_terms"] = [((None, None, b), env) for b, env in terms[1:]]
    if c["damp"]:
        opts["vel_damp"] = c["damp"]
    if c["kahan"]:
        opts["kahan"] = True
    return dict(bx=None, by=None, bz=terms[0][0], rho=rho, mu=mu, dX=H, dY=H, dZ=H, dT=dT,
                n_steps=n, opts=opts)


def _batch_cases(c, seed):
    """The solves of a batch: grids and lengths from the case alone, values from the seed."""
    rng = np.random.default_rng(c["count"] * 7919 + c["hi"] * 31 + c["steps_hi"])
    out = []
    for k in range(c["count"]):
        nx, ny = (int(v) for v in rng.integers(c["lo"], c["hi"] + 1, 2))
        nz = int(rng.integers(c["lo"], c["hi_z"] + 1))
        n = int(rng.integers(c["steps_lo"], c["steps_hi"] + 1))
        out.append((dict(nx=nx, ny=ny, nz=nz, n_steps=n, precision=c["precision"],
                         medium="inclusions", eta="map", pushes=1, damp=0.0, stride=0,
                         kahan=False), seed * 1000 + k))
    return out


def _forces(c, seed):
    rng = np.random.default_rng(seed)
    shape, dtype = (c["nx"], c["ny"], c["nz"]), getattr(torch, c["dtype"])
    size = np.array(shape) * H
    comps = []
    for k in range(3):
        if k < 3 - c["comps"]:
            comps.append(torch.zeros(shape, device=DEV, dtype=dtype))
            continue
        centre = (0.25 + 0.5 * rng.uniform(0.0, 1.0, 3)) * size
        comps.append(_push(shape, centre, 1.5e-3, 5e-3, dtype, 1e3 * rng.uniform(0.5, 1.5)))
    return comps


def _displacement(shape, seed, dtype):
    """(nx, ny, nz, 3) displacement of shear waves of 4-12 mm [m], zero shell."""
    rng, gen = np.random.default_rng(seed), _gen(seed)
    u = torch.stack([_smooth(shape, rng, gen) for _ in range(3)], dim=-1) * 1e-5
    out = torch.zeros_like(u)
    out[1:-1, 1:-1, 1:-1] = u[1:-1, 1:-1, 1:-1]
    return out.to(dtype)


def _records(c, seed):
    """Recorded tone burst: pressure [Pa], and velocities [m/s] for the vector form."""
    rng, gen = np.random.default_rng(seed), _gen(seed)
    shape, nt, dtype = (c["nx"], c["ny"], c["nz"]), c["nt"], getattr(torch, c["dtype"])
    centre = np.array(shape) * H * (0.3 + 0.4 * rng.uniform(0.0, 1.0, 3))
    beam = _push(shape, centre, 4e-3, 10e-3, torch.float64, 1e6).reshape(-1, 1)
    t = torch.arange(nt, device=DEV, dtype=torch.float64)
    burst = torch.exp(-0.5 * ((t - 0.45 * nt) / (0.12 * nt)) ** 2)
    fields = []
    for k in range(4 if c["velocity"] else 1):
        scale = 1.0 if k == 0 else (6e-7 if k == 3 else 1e-7)
        phase = float(rng.uniform(0, 2 * math.pi))
        wave = (burst * torch.sin(0.7 * t + phase))[None, :]
        f = torch.randn((beam.shape[0], nt), generator=gen, device=DEV, dtype=torch.float32)
        f = f.to(dtype) * (2e3 * scale)
        f += ((beam * scale).to(dtype)) * wave.to(dtype)
        fields.append(f.reshape(*shape, nt))
    if c["maps"]:
        maps = [(v * (1.0 + 0.05 * _smooth(shape, rng, gen))).to(dtype)
                for v in (1540.0, 1000.0, 0.5)]
    else:
        maps = [1540.0, 1000.0, 0.5]
    gate = None
    if c["gate"] == "slice":
        gate = slice(nt // 4, nt - nt // 4)
    elif c["gate"] == "mask":
        gate = np.zeros(nt, bool)
        gate[nt // 5: nt - nt // 5: 2] = True
    return fields, maps, gate


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "solve":
        return dict(kind=kind, args=_problem(c, seed), stride=c["stride"] or None)
    if kind == "batch":
        return dict(kind=kind, args=[_problem(k, s) for k, s in _batch_cases(c, seed)])
    if kind == "project":
        return dict(kind=kind, f=_forces(c, seed), tol=c["tol"], iters=c["iters"],
                    method=c["method"])
    shape = (c["nx"], c["ny"], c["nz"])
    dtype = getattr(torch, c["dtype"])
    if kind == "static":
        rng, gen = np.random.default_rng(seed), _gen(seed)
        centre = (0.3 + 0.4 * rng.uniform(0.0, 1.0, 3)) * np.array(shape) * H
        mu = 2000.0 * float(rng.uniform(0.8, 1.2))
        if c["field"]:
            mu = (mu * (1.0 + 0.1 * _smooth(shape, rng, gen))).to(dtype)
        return dict(kind=kind, b=_push(shape, centre, 1.5e-3, 5e-3, dtype), mu=mu, tol=c["tol"],
                    iters=c["iters"])
    if kind == "strain":
        u = _displacement(shape, seed, dtype)
        if c["form"] == "tensor":
            return dict(kind=kind, form=c["form"], u=[u[..., k].contiguous() for k in range(3)])
        return dict(kind=kind, form=c["form"], u=u)
    if kind == "arf":
        fields, maps, gate = _records(c, seed)
        return dict(kind=kind, fields=fields, maps=maps, gate=gate)
    u = _displacement(shape, seed, dtype)
    return dict(kind=kind, u=[u[..., k].contiguous() for k in range(3)])


def run(state):
    kind = state["kind"]
    if kind == "solve":
        return sw.shear_fdtd(**state["args"], snapshot_stride=state["stride"],
                             return_device=True)
    if kind == "batch":
        return sw.shear_fdtd_batch(state["args"], return_device=True)
    if kind == "project":
        return sw.project_vector_field(*state["f"], H, H, H, state["tol"], state["iters"],
                                       method=state["method"])
    if kind == "static":
        return sw.elastic_solve_static(state["b"], H, H, H, state["mu"], state["tol"],
                                       state["iters"])
    if kind == "strain":
        if state["form"] == "tensor":
            eps = sw.compute_strain_tensor(*state["u"], H, H, H)
            return eps, sw.compute_strain_invariants(eps)
        return sw.compute_strain_fields(state["u"], H, H, H,
                                        return_tensor=state["form"] == "fields",
                                        return_device=True)
    if kind == "arf":
        call = (sw.compute_radiation_force if len(state["fields"]) == 1
                else sw.compute_radiation_force_velocity)
        return call(*state["fields"], *state["maps"], 5e6, gate=state["gate"])
    ux, uy, uz = state["u"]
    return (sw.laplacian_center(uz, H, H, H), sw.divergence_center(ux, uy, uz, H, H, H),
            sw.gradient_center(uz, H, H, H))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _solve_work(c):
    """Inputs and outputs once; per cell and step three components of two
    seven-point Laplacians (one without viscosity) and the update."""
    n = c["nx"] * c["ny"] * c["nz"]
    es = 8 if c["precision"] == "fp64" else 4
    maps = (0 if c["medium"] == "uniform" else 2) + (1 if c["eta"] == "map" else 0)
    snaps = c["n_steps"] // c["stride"] if c["stride"] else 0
    per = 3 * ((13 if c["eta"] == "none" else 26) + (1 if c["damp"] else 0))
    return es * n * (maps + c["pushes"] + 6 + 3 * snaps), float(per) * n * c["n_steps"]


def work(case):
    c = dict(case)
    kind = c["kind"]
    if kind == "solve":
        b, f = _solve_work(c)
        return {"bytes": b, "flops": f}
    if kind == "batch":
        both = [_solve_work(k) for k, _ in _batch_cases(c, 0)]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    n = c["nx"] * c["ny"] * c["nz"]
    es = 4 if c["dtype"] == "float32" else 8
    if kind == "project":
        # the direct solve's six one-axis transforms, each on two half-length chains
        return {"bytes": 6 * es * n, "flops": 2.0 * n * (c["nx"] + c["ny"] + c["nz"])}
    if kind == "static":
        return {"bytes": (3 if c["field"] else 2) * es * n,
                "flops": 4.0 * n * (c["nx"] + c["ny"] + c["nz"])}
    if kind == "strain":
        out = (6 if c["form"] != "invariants" else 0) * es + 3 * es + 8
        return {"bytes": n * (3 * es + out), "flops": 45.0 * n}
    if kind == "arf":
        k = 4 if c["velocity"] else 1
        return {"bytes": n * es * ((k if c["gate"] != "auto" else 1) * c["nt"]
                                   * (0.5 if c["gate"] == "slice" else 1.0)
                                   + (3 if c["maps"] else 0) + (3 if c["velocity"] else 1)),
                "flops": 2.0 * n * c["nt"]}
    return {"bytes": es * n * (3 + 1 + 1 + 3), "flops": 30.0 * n}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
_I = (slice(1, -1),) * 3


def _nb(f, axis, k):
    """Interior cells of f moved by k along an axis."""
    sl = [slice(1, -1)] * 3
    sl[axis] = slice(1 + k, f.shape[axis] - 1 + k)
    return f[tuple(sl)]


def _lap(f):
    out = torch.zeros_like(f)
    out[_I] = sum(_nb(f, a, 1) + _nb(f, a, -1) for a in range(3)).sub_(f[_I], alpha=6.0) / (H * H)
    return out


def _div(comps):
    out = torch.zeros_like(comps[0])
    out[_I] = sum((_nb(f, a, 1) - _nb(f, a, -1)) / (2 * H) for a, f in enumerate(comps))
    return out


def _grad(f):
    outs = []
    for a in range(3):
        g = torch.zeros_like(f)
        g[_I] = (_nb(f, a, 1) - _nb(f, a, -1)) / (2 * H)
        outs.append(g)
    return outs


def _masked(f):
    out = torch.zeros_like(f)
    out[_I] = f[_I]
    return out


def _cg(apply, b, tol, iters, projection):
    """The reference's conjugate gradient and stopping rule."""
    eps = 2.220446049250313e-16
    x, r, p = torch.zeros_like(b), b.clone(), b.clone()
    rs = float((r * r).sum())
    rs0 = max(rs, eps) if projection else rs + 1e-30
    for _ in range(iters):
        ap = apply(p)
        pap = float((p * ap).sum())
        if not math.isfinite(pap) or pap <= 0.0:
            break
        alpha = rs / pap
        x.add_(p, alpha=alpha)
        r.sub_(ap, alpha=alpha)
        new = float((r * r).sum())
        if not math.isfinite(new) or math.sqrt(new / rs0) < tol:
            break
        p.mul_(new / max(rs, eps)).add_(r)
        rs = new
    return x


def _project(comps, tol, iters, direct):
    comps = [_masked(f.double()) for f in comps]
    rhs = -_div(comps)
    if direct:
        b, lams, qs = rhs[_I], [], []
        for n in rhs.shape:
            g = torch.zeros((n, n), device=rhs.device, dtype=torch.float64)
            i = torch.arange(1, n - 1, device=rhs.device)
            g[i, i + 1], g[i, i - 1] = 1 / (2 * H), -1 / (2 * H)
            lam, q = torch.linalg.eigh(-(g @ g)[1:-1, 1:-1])
            lams.append(lam)
            qs.append(q)
        for a in range(3):
            b = torch.tensordot(b, qs[a], dims=([0], [0]))  # the axes turn round once
        total = lams[0][:, None, None] + lams[1][None, :, None] + lams[2][None, None, :]
        b = torch.where(total > 1e-13 * 12 / (H * H), b / total, 0.0)
        for a in range(3):
            b = torch.tensordot(b, qs[a].T, dims=([0], [0]))
        phi = torch.zeros_like(rhs)
        phi[_I] = b
    else:
        phi = _cg(lambda v: -_div(_grad(v)), rhs, tol, iters, True)
    return [_masked(f - g) for f, g in zip(comps, _grad(phi))]


def _solve_exact(p, stride):
    o = p["opts"]
    n, dT = p["n_steps"], p["dT"]
    shape = tuple(p["bz"].shape)

    def field(v):
        return v.double() if isinstance(v, torch.Tensor) else float(v)

    rho, mu, eta = field(p["rho"]), field(p["mu"]), field(o["eta"])
    m, e = dT * dT * mu / rho, dT * eta / rho
    viscous = isinstance(eta, torch.Tensor) or eta != 0.0
    fp64 = o["precision"] == "fp64"
    terms = [(p["bz"], o["env_t"])] + [(t[0][2], t[1]) for t in o.get("force_terms") or ()]
    zero = torch.zeros(shape, device=DEV, dtype=torch.float64)
    pats = []
    for b, env in terms:
        f = _project([zero, zero, b], 1e-10, o["poisson_max_iters"], not fp64)
        pats.append((torch.stack(f) * (dT * dT) / rho, env))
    inner = (slice(None), *_I)

    def sub(f, axis, k):
        sl = [slice(None)] + [slice(1, -1)] * 3
        sl[1 + axis] = slice(1 + k, f.shape[1 + axis] - 1 + k)
        return f[tuple(sl)]

    def lap(f, out):
        torch.add(sub(f, 0, 1), sub(f, 0, -1), out=out)
        for a, k in ((1, 1), (1, -1), (2, 1), (2, -1)):
            out.add_(sub(f, a, k))
        return out.add_(f[inner], alpha=-6.0)

    u = torch.zeros((3, *shape), device=DEV, dtype=torch.float64)
    d = torch.zeros_like(u)
    mi = (m[_I] if isinstance(m, torch.Tensor) else m) / (H * H)
    ei = (e[_I] if isinstance(e, torch.Tensor) else e) / (H * H)
    w, w2 = torch.empty_like(u[inner]), torch.empty_like(u[inner])
    damp = 1.0 - o.get("vel_damp", 0.0)
    snaps = []
    for it in range(n):
        lap(u, w).mul_(mi)
        if viscous:
            w.add_(lap(d, w2).mul_(ei))
        di = d[inner]
        di.add_(w)
        for pat, env in pats:
            if env[it] != 0.0:
                di.add_(pat[inner], alpha=float(env[it]))
        if damp != 1.0:
            di.mul_(damp)
        u[inner] += di
        if stride and (it + 1) % stride == 0:
            snaps.append(u.permute(1, 2, 3, 0).contiguous())
    out = [u.permute(1, 2, 3, 0).contiguous(), (d / dT).permute(1, 2, 3, 0).contiguous()]
    if stride:
        out.append(torch.stack(snaps))
    return tuple(out)


def _invariants(eps):
    vol = eps[..., :3].sum(-1) / 3.0
    dev = eps[..., :3] - vol[..., None]
    s = (dev * dev).sum(-1) + 0.5 * (eps[..., 3:] ** 2).sum(-1)
    return dict(volumetric=vol, deviatoric=s.sqrt(), max_shear=(0.5 * s).sqrt(),
                von_mises=math.sqrt(2.0 / 3.0) * s.sqrt())


def _strain_exact(comps):
    g = [_grad(f.double()) for f in comps]
    return torch.stack([g[0][0], g[1][1], g[2][2], g[1][2] + g[2][1], g[0][2] + g[2][0],
                        g[0][1] + g[1][0]], dim=-1)


def _arf_exact(fields, maps, gate):
    p = fields[0]
    nt = p.shape[-1]
    if gate is None:
        total = torch.zeros(nt, device=DEV, dtype=torch.float64)
        for plane in p:
            total += plane.double().square().sum((0, 1))
        idx = torch.nonzero(total >= 0.1 * total.max())[:, 0]
    else:
        idx = torch.as_tensor(np.arange(nt)[gate], device=DEV)
    c, rho, alpha = (m.double() if isinstance(m, torch.Tensor) else m for m in maps)
    alpha_np = alpha * 5.0 / 8.685889638 * 100.0
    outs = []
    for q in fields if len(fields) == 1 else fields[1:]:
        mean = torch.stack([(a[..., idx].double() * b[..., idx].double()).mean(-1)
                            for a, b in zip(p, q)])
        if len(fields) == 1:
            return 2.0 * alpha_np * (mean / (rho * c)) / c
        outs.append(2.0 * alpha_np / c * mean)
    return tuple(outs)


def exact(case, seed):
    c = dict(case)
    s = prepare(c, seed)
    kind = c["kind"]
    if kind == "solve":
        return _solve_exact(s["args"], s["stride"])
    if kind == "batch":
        return [_solve_exact(p, None) for p in s["args"]]
    if kind == "project":
        return tuple(_project(s["f"], s["tol"], s["iters"], s["method"] == "spectral"))
    if kind == "static":
        mu = s["mu"].double() if isinstance(s["mu"], torch.Tensor) else s["mu"]
        return _cg(lambda v: -mu * _lap(v), _masked(s["b"].double()), s["tol"], s["iters"], False)
    if kind == "strain":
        u = s["u"] if c["form"] == "tensor" else [s["u"][..., k] for k in range(3)]
        eps = _strain_exact(u)
        return (None if c["form"] == "invariants" else eps), _invariants(eps)
    if kind == "arf":
        return _arf_exact(s["fields"], s["maps"], s["gate"])
    ux, uy, uz = (f.double() for f in s["u"])
    return _lap(uz), _div([ux, uy, uz]), tuple(_grad(uz))

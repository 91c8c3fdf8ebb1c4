"""The work that users of illum_gb300 have it do, as measurable cases.

Each case is one way into the package: a set-up call made once per shape model
(LBVH, horizon maps, form factors), a solver called by itself, or the time-step
loop over a whole body, over the sizes, boundaries and precisions of the
benchmark configurations, from the smallest mesh to the large terrain.

``listed()`` are the fixed cases, ``draw(rng)`` gives further ones of the same
ranges. ``prepare`` makes what a program holds before the call, ``run`` is one
call, ``work`` the bytes and operations that call cannot do without, and
``exact`` its result in plain 64-bit numpy or torch where that is affordable.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import illum_gb300 as ig
from illum_gb300 import meshgen

SIGMA = 5.6704e-8      # W m^-2 K^-4, the value of the conduction routines
SOLAR = 1361.0
RHOC = 1500.0 * 700.0
ALBEDO = 0.1

# Shape models: icosphere level -> craters (count, smallest and largest
# diameter in m): the 5,120-facet and 81,920-facet configurations, and the
# batched workload's crater rate in between.
CRATERS = {3: (6, 80.0, 300.0), 4: (20, 80.0, 300.0), 5: (50, 30.0, 300.0), 6: (200, 30.0, 300.0)}


def _facets(c):
    if c.get("terrain"):
        return 2 * (c["terrain"] - 1) ** 2
    return 20 * 4 ** c["level"]


def listed():
    return [
        # conductionQ called with arrays of columns (the drop-in Fortran path,
        # batched): one small body's worth of columns
        {"name": "columns", "kind": "columns", "ncol": 5120, "nz": 40, "bc": 1},
        # one time step with the sun position from the host and the surface
        # temperatures back: a program that follows an ephemeris step by step
        {"name": "live_step", "kind": "live", "level": 4, "nz": 40, "steps": 1},
        # radiosity alone for a form-factor matrix from a file, to tolerance
        {"name": "solve", "kind": "solve", "level": 6, "cutoff_m": 150.0, "method": "tol"},
        # the same with the reference's fixed Gauss-Seidel sweeps (the command
        # line's default solve)
        {"name": "solve_gs", "kind": "solve", "level": 6, "cutoff_m": 150.0, "method": "gs"},
        # set-up of a new shape model: LBVH, horizon map and form factors, as
        # the serving loop does for every request
        {"name": "setup", "kind": "setup", "level": 5, "nphi": 32, "smooth": True, "shape": 11},
        # horizon map of the 81,920-facet body
        {"name": "horizons", "kind": "horizons", "level": 6, "nphi": 64},
        # form factors of a terrain patch within a distance cutoff
        {"name": "terrain_F", "kind": "terrain_F", "terrain": 256, "cutoff_m": 30.0, "shape": 7},
        # the 81,920-facet body, an eighth of a rotation in FP64, and a
        # quarter of a rotation in mixed precision
        {"name": "steps_fp64", "kind": "steps", "level": 6, "nz": 60, "steps": 90, "mixed": False},
        {"name": "steps_mixed", "kind": "steps", "level": 6, "nz": 60, "steps": 180, "mixed": True},
        # many bodies of mixed sizes and depths stepped together
        {"name": "batch_mixed", "kind": "batch", "meshes": 16, "top": 6, "steps": 60, "mixed": True},
        {"name": "batch_fp64", "kind": "batch", "meshes": 16, "top": 6, "steps": 20, "mixed": False},
        # a large terrain patch, radiosity refined to 1e-8 of the flux: the
        # largest matrix, far beyond L2
        {"name": "terrain_mixed", "kind": "terrain", "terrain": 512, "cutoff_m": 30.0, "nz": 40, "steps": 4},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["columns", "live", "solve", "solve", "setup", "horizons", "terrain_F", "steps", "steps",
                       "batch", "batch", "terrain"])
    c = {"kind": kind}
    if kind == "columns":
        c["ncol"] = int(_log(rng, 64, 82000))
        c["nz"] = rng.randint(30, 80)
        c["bc"] = rng.choice([0, 1])
    elif kind == "live":
        c.update(level=rng.choice([3, 4, 5, 6]), nz=rng.randint(30, 80), steps=rng.randint(1, 5))
    elif kind == "solve":
        c.update(level=rng.choice([4, 5, 6]), cutoff_m=round(rng.uniform(50.0, 150.0), 1),
                 method=rng.choice(["tol", "tol", "gs"]))
    elif kind == "setup":
        c.update(level=rng.choice([3, 4, 5]), nphi=rng.choice([32, 33, 64, 91]), smooth=rng.random() < 0.7,
                 shape=rng.randrange(1 << 20))
    elif kind == "horizons":
        c.update(level=rng.choice([4, 5, 6]), nphi=rng.choice([32, 48, 61, 64]))
    elif kind == "terrain_F":
        c.update(terrain=int(_log(rng, 64, 256)), cutoff_m=round(rng.uniform(12.0, 30.0), 1),
                 shape=rng.randrange(1 << 20))
    elif kind == "steps":
        c.update(level=rng.choice([4, 5, 6]), nz=rng.randint(30, 80), steps=rng.choice([20, 37, 60, 90]),
                 mixed=rng.random() < 0.5)
    elif kind == "batch":
        c.update(meshes=rng.randint(2, 16), top=rng.choice([4, 5, 6]), steps=rng.choice([10, 20, 30]),
                 mixed=rng.random() < 0.5)
    else:
        c.update(terrain=int(_log(rng, 128, 512)), cutoff_m=round(rng.uniform(12.0, 30.0), 1), nz=rng.randint(30, 60),
                 steps=rng.randint(1, 4))
    return c


# ------------------------------------------------------------------ inputs
def _mesh(level, seed, smooth=False):
    n, dmin, dmax = CRATERS[level]
    return meshgen.icosphere_craters(level, seed, sigma_m=0.0 if smooth else 15.0, n_craters=n, dmin_m=dmin,
                                     dmax_m=dmax)


def _terrain_mesh(c, seed):
    n = c["terrain"]
    return meshgen.heightmap_terrain(n=n, spacing_m=2.0, seed=seed, n_bowls=max(1, 2000 * n * n // (1024 * 1024)),
                                     dmin_m=10.0, dmax_m=min(400.0, 0.8 * n))


def _surface(c, mesh, seed):
    """The case's shape with what the seed gives: the face its list begins
    with (every facet index changes), and an albedo map. (How many facets see
    each other is the shape's, so the matrix has one size per case.)"""
    v, f = mesh
    g = np.random.default_rng(seed)
    return v, np.roll(f, int(g.integers(1, f.shape[0])), axis=0), g.uniform(0.04, 0.16, f.shape[0])


def _material(seed, k=0):
    """Thermal inertia (log-uniform 50-2000 SI), rotation period (2-12 h)."""
    u = meshgen.uniform(seed + 7919 * k, 21, 2)
    return float(50.0 * 40.0 ** u[0]), float(3600.0 * (2.0 + 10.0 * u[1]))


def _body(level, seed, nphi, rad_blocks=False):
    v, f = _mesh(level, seed)
    ctx = ig.IllumContext(v, f)
    ctx.make_horizons(nphi=nphi)
    ctx.set_insolation(1, 0, SOLAR)
    ctx.compute_F(albedo=ALBEDO, fetch=False)
    if rad_blocks:   # stepped beside other bodies: tiles for the batch, not for one body alone
        ctx.set_radiosity_blocks(ig.radiosity_blocks_for(ctx.F_info()["nnz"]))
    return ctx


def _thermal(ctx, nz, ti, mixed):
    return ig.ThermalModel(ctx, meshgen.geometric_depths(nz), ti, RHOC, 200.0, emissivity=0.95,
                           bc_mode=ig.BC_NEWTON, precision=ig.PREC_MIXED if mixed else ig.PREC_FP64)


def _opts(dt, mixed, refine_every=4):
    if mixed:
        return ig.RunOpts(dt=dt, tol=1e-3, max_sweeps=1, use_radiosity=1, use_graph=1, precision=ig.PREC_MIXED,
                          coupling=ig.COUPLE_DIRECT, refine_every=refine_every)
    return ig.RunOpts(dt=dt, tol=1e-10, max_sweeps=200, use_radiosity=1, use_graph=1, precision=ig.PREC_FP64,
                      coupling=ig.COUPLE_DIRECT)


def _columns_inputs(c, seed):
    """Columns of a body mid-way through a day: skin temperatures between
    night and noon, relaxing to a common value at depth."""
    g = np.random.default_rng(seed)
    ncol, nz = c["ncol"], c["nz"]
    z = meshgen.geometric_depths(nz)
    ts = g.uniform(90.0, 320.0, ncol)
    deep = g.uniform(180.0, 220.0, ncol)
    T = np.asfortranarray(deep[None, :] + (ts - deep)[None, :] * np.exp(-z / 0.05)[:, None]
                          + g.normal(0.0, 0.05, (nz, ncol)))
    Q = np.maximum(0.0, g.uniform(-300.0, 600.0, ncol))
    Qn = np.maximum(0.0, Q + g.normal(0.0, 5.0, ncol))
    ti = np.full(nz, float(50.0 * 40.0 ** g.uniform()))
    return dict(z=z, dt=float(g.uniform(30.0, 60.0)), Qn=Qn, Qnp1=Q, T=T, ti=ti, rhoc=np.full(nz, RHOC), emiss=0.95,
                Tsurf=ts)


def _matrix(c, seed):
    """Form factors as a file holds them (CSR by receiver row): every pair of
    facets of a cratered body that face each other within a distance, with
    the point-to-point form factor and the albedo; and a flux at some hour."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    v, f = _mesh(c["level"], seed)
    V = torch.tensor(v, dtype=torch.float64, device=dev)
    F = torch.tensor(f, dtype=torch.int64, device=dev)
    a, b, d = V[F[:, 0]], V[F[:, 1]], V[F[:, 2]]
    cr = torch.linalg.cross(b - a, d - a)
    area = 0.5 * cr.norm(dim=1)
    n = cr / (2.0 * area)[:, None]
    p = (a + b + d) / 3.0
    N = p.shape[0]
    cut = c["cutoff_m"] / 1000.0
    rows, cols, vals = [], [], []
    for r0 in range(0, N, 1024):
        r1 = min(N, r0 + 1024)
        w = p[None, :, :] - p[r0:r1, None, :]
        r2 = (w * w).sum(-1)
        mi = (w * n[r0:r1, None, :]).sum(-1)
        mj = -(w * n[None, :, :]).sum(-1)
        ok = (r2 > 0) & (r2 <= cut * cut) & (mi > 0) & (mj > 0)
        i, j = ok.nonzero(as_tuple=True)
        rows.append(i + r0)
        cols.append(j)
        vals.append(ALBEDO * mi[i, j] * mj[i, j] * area[j] / (math.pi * r2[i, j] ** 2))
    rows, cols, vals = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    rowptr = torch.zeros(N + 1, dtype=torch.int64, device=dev)
    rowptr[1:] = torch.bincount(rows, minlength=N).cumsum(0)
    u = np.random.default_rng(seed).normal(size=3)
    sun = torch.tensor(u / np.linalg.norm(u), device=dev)
    E = 600.0 * torch.clamp((n * sun).sum(1), min=0.0)
    return v, f, rowptr.cpu().numpy(), cols.to(torch.int32).cpu().numpy(), vals.cpu().numpy(), E.cpu().numpy()


def prepare(case, seed):
    c, k = case, case["kind"]
    s = {"case": c, "sun": 0}
    if k == "columns":
        s["in"] = _columns_inputs(c, seed)
    elif k == "solve":
        v, f, rowptr, col, val, E = _matrix(c, seed)
        s["ctx"] = ctx = ig.IllumContext(v, f)
        ctx.set_F(rowptr, col, val)
        s["E"] = E
    elif k == "setup":
        s["v"], s["f"], s["albedo"] = _surface(c, _mesh(c["level"], c["shape"], smooth=c["smooth"]), seed)
    elif k == "horizons":
        s["ctx"] = ig.IllumContext(*_mesh(c["level"], seed))
    elif k == "terrain_F":
        v, f, s["albedo"] = _surface(c, _terrain_mesh(c, c["shape"]), seed)
        s["ctx"] = ig.IllumContext(v, f)
    elif k == "live":
        ti, period = _material(seed)
        s["ctx"] = ctx = _body(c["level"], seed, 32)
        s["suns"] = meshgen.spin_sun_positions(360, period, period / 360)
        ctx.set_suns(s["suns"][:1], ig.fib_spiral(100))   # the disk samples; the positions come step by step
        s["tm"] = _thermal(ctx, c["nz"], ti, False)
        s["opts"] = _opts(period / 360, False)
    elif k == "steps":
        ti, period = _material(seed)
        s["ctx"] = ctx = _body(c["level"], seed, 64 if c["level"] == 6 else 32)
        ctx.set_suns(meshgen.spin_sun_positions(720, period, period / 720), ig.fib_spiral(100))
        s["nsun"] = 720
        s["tm"] = _thermal(ctx, c["nz"], ti, c["mixed"])
        s["opts"] = _opts(period / 720, c["mixed"])
    elif k == "terrain":
        v, f = _terrain_mesh(c, seed)
        ti, period = _material(seed)
        s["ctx"] = ctx = ig.IllumContext(v, f)
        ctx.make_horizons(nphi=128)
        ctx.set_insolation(1, 0, SOLAR)
        ctx.compute_F(albedo=ALBEDO, cutoff=c["cutoff_m"] / 1000.0, fetch=False)
        # the daylight quarter before and after noon, again and again
        suns = np.concatenate([meshgen.site_sun_positions(72, period, period / 360),
                               meshgen.site_sun_positions(72, period, period / 360, t0_s=-period / 5)])
        ctx.set_suns(suns, ig.fib_spiral(100))
        s["nsun"] = 144
        s["tm"] = _thermal(ctx, c["nz"], ti, True)
        o = _opts(period / 360, True, refine_every=0)
        o.tol = 1e-8 * 500.0 * math.sqrt(_facets(c))   # 1e-8 of the 2-norm of the daytime flux
        o.max_sweeps = 400
        s["opts"] = o
    elif k == "batch":
        s["members"], s["tms"], opts = [], [], []
        for m in range(c["meshes"]):
            ti, period = _material(seed, m)
            ctx = _body(c["top"] - m % 4 if c["top"] - m % 4 >= 3 else 3, seed * 64 + m, 32, rad_blocks=True)
            # a batch's members run off the end of their sun tables: many rotations
            ctx.set_suns(meshgen.spin_sun_positions(1 << 16, period, period / 360), ig.fib_spiral(100))
            s["tms"].append(_thermal(ctx, 30 + (m * 37) % 51, ti, c["mixed"]))
            s["members"].append(ctx)
            opts.append(_opts(period / 360, c["mixed"]))
        s["batch"] = ig.Batch(s["members"], opts)
    return s


# ------------------------------------------------------------------ the call
def _keep(out, mixed):
    """Mixed-precision results are kept in the 32 bits they are good for."""
    return {k: a.astype(np.float32) for k, a in out.items()} if mixed else out


def run(state):
    s, c = state, state["case"]
    k = c["kind"]
    if k == "columns":
        T, ts, fs = ig.conductionQ_batch(bc_mode=c["bc"], **s["in"])
        return {"T": T, "Tsurf": ts, "Fsurf": fs}
    if k == "solve":
        if c["method"] == "gs":
            x, _ = s["ctx"].radiosity_solve_gs(s["E"], gs_steps=1)
        else:
            x, _, _ = s["ctx"].radiosity_solve(s["E"], tol=1e-10)
        return x
    if k == "setup":
        ctx = ig.IllumContext(s["v"], s["f"])
        ctx.make_horizons(nphi=c["nphi"])
        rowptr, col, val = ctx.compute_F(albedo=s["albedo"])
        H = ctx.horizons
        ctx.close()
        return {"H": H, "rowptr": rowptr, "col": col, "val": val}
    if k == "horizons":
        s["ctx"].make_horizons(nphi=c["nphi"])
        return s["ctx"].horizons
    if k == "terrain_F":
        rowptr, col, val = s["ctx"].compute_F(albedo=s["albedo"], cutoff=c["cutoff_m"] / 1000.0)
        return {"rowptr": rowptr, "col": col, "val": val}
    if k == "live":
        at = (s["sun"] + np.arange(c["steps"])) % s["suns"].shape[0]
        s["sun"] += c["steps"]
        return s["ctx"].run_steps_host(s["opts"], s["suns"][at])
    if k == "batch":
        s["batch"].run(c["steps"])
        return _keep({str(m): s["batch"].tsurf(m) for m in range(c["meshes"])}, c["mixed"])
    # steps, terrain
    if s["sun"] + c["steps"] > s["nsun"]:
        s["sun"] = 0
    s["ctx"].run_steps(s["opts"], s["sun"], c["steps"])
    s["sun"] += c["steps"]
    out = s["ctx"].outputs()
    out["Fsurf"] = s["tm"].get_F()
    return _keep(out, k == "terrain" or c["mixed"])


# ------------------------------------------------------------------ its work
def _pairs(level):
    """Form-factor entries of a cratered body: facets of a crater see most of
    the others of the same crater."""
    n, a, b = CRATERS[level]
    N = 20 * 4 ** level
    d4 = (b ** 5 - a ** 5) / (5.0 * (b - a))          # mean of the diameter's fourth power
    return 0.9 * n * d4 * (N / 16e6) ** 2


def _terrain_pairs(c):
    return _facets(c) * 195.0 * (c["cutoff_m"] / 30.0) ** 1.55


def _step_work(N, nz, nnz, mixed):
    """One step: every layer read and written, the facet's scalars, the
    matrix once, the disk test of each facet."""
    layer, entry = (4, 4) if mixed else (8, 10)
    return N * (2.0 * nz * layer + 12 * 8) + nnz * entry, N * (nz * 12.0 + 200.0) + 2.0 * nnz


def work(case):
    c, k = case, case["kind"]
    if k == "columns":
        n, nz = c["ncol"], c["nz"]
        return {"bytes": 8.0 * n * (2 * nz + 5), "flops": 14.0 * n * nz + 60.0 * n}
    N = _facets(c) if k != "batch" else 0
    if k == "solve":
        nnz = 2.7e5 * 16.0 ** (c["level"] - 5) * (c["cutoff_m"] / 100.0) ** 1.5
        return {"bytes": 12.0 * nnz + 24.0 * N, "flops": 2.0 * nnz * (3 if c["method"] == "gs" else 6)}
    if k in ("setup", "horizons"):
        # one ray per azimuth and bisection level, one per facing pair (about
        # a tenth of all), each down a tree of log2 N levels to one triangle
        rays = 11.0 * N * c["nphi"]
        out = 8.0 * N * c["nphi"]
        if k == "setup":
            rays += 0.1 * N * N
            out += 12.0 * _pairs(c["level"]) + 8.0 * N
        return {"bytes": out + 24.0 * N, "flops": rays * (math.log2(N) * 24.0 + 40.0)}
    if k == "terrain_F":
        nnz = _terrain_pairs(c)
        return {"bytes": 12.0 * nnz + 32.0 * N, "flops": 4.0 * nnz * (math.log2(N) * 24.0 + 40.0)}
    if k == "batch":
        b = f = 0.0
        for m in range(c["meshes"]):
            level = max(3, c["top"] - m % 4)
            x, y = _step_work(20 * 4 ** level, 30 + (m * 37) % 51, _pairs(level), c["mixed"])
            b, f = b + x, f + y
    else:
        mixed = c.get("mixed", k == "terrain")
        b, f = _step_work(N, c["nz"], _terrain_pairs(c) if k == "terrain" else _pairs(c["level"]), mixed)
    return {"bytes": b * c["steps"], "flops": f * c["steps"]}


# ------------------------------------------------------------------ in 64 bits
def _exact_columns(c, seed):
    """Crank-Nicolson in numpy: T at the new time is affine in the surface
    temperature, so two tridiagonal solves and a scalar root."""
    q = _columns_inputs(c, seed)
    z, dt, T, ti, rhoc = q["z"], q["dt"], np.array(q["T"]), q["ti"], q["rhoc"]
    nz = z.shape[0]
    cond = ti * ti / rhoc
    al, ga = np.zeros(nz), np.zeros(nz)
    h = 2.0 * z[0]
    al[0] = dt / rhoc[0] / (2.0 * h * h) * cond[1]
    ga[0] = dt / rhoc[0] / (2.0 * h * h) * cond[0]
    for i in range(1, nz - 1):
        w = dt / (z[i + 1] - z[i - 1])
        al[i] = 2.0 * cond[i + 1] * w / (rhoc[i] + rhoc[i + 1]) / (z[i + 1] - z[i])
        ga[i] = 2.0 * cond[i] * w / (rhoc[i] + rhoc[i + 1]) / (z[i] - z[i - 1])
    ga[-1] = cond[-1] * dt / (z[-1] - z[-2]) ** 2 / (2.0 * rhoc[-1])
    k1, es, Ts, Qn, Q = cond[0] / h, q["emiss"] * SIGMA, q["Tsurf"], q["Qn"], q["Qnp1"]
    R = np.empty_like(T)
    R[1:-1] = ga[1:-1, None] * T[:-2] + (1.0 - al - ga)[1:-1, None] * T[1:-1] + al[1:-1, None] * T[2:]
    R[-1] = ga[-1] * T[-2] + (1.0 - ga[-1]) * T[-1]
    if c["bc"] == 1:
        b0 = np.full(T.shape[1], 1.0 + al[0] + 2.0 * ga[0])
        R[0] = (1.0 - al[0] - ga[0]) * T[0] + al[0] * T[1] + ga[0] * (2.0 * Ts - T[0])
    else:
        ar, br = -3.0 * es * Ts ** 4, 2.0 * es * Ts ** 3
        den = k1 + br
        an, an1, bn = (Qn - ar) / den, (Q - ar) / den, (k1 - br) / den
        b0 = 1.0 + al[0] + ga[0] - ga[0] * bn
        R[0] = ga[0] * (an + an1) + (1.0 - al[0] - ga[0] + ga[0] * bn) * T[0] + al[0] * T[1]
    # from the bottom: each layer in terms of the one above it
    r, b = np.empty_like(T), np.empty(nz)
    b[-1], r[-1] = 1.0 + ga[-1], R[-1]
    for i in range(nz - 2, 0, -1):
        m = al[i] / b[i + 1]
        b[i] = 1.0 + al[i] + ga[i] - m * ga[i + 1]
        r[i] = R[i] + m * r[i + 1]
    m = al[0] / b[1]
    top, rt = b0 - m * ga[1], R[0] + m * r[1]
    if c["bc"] == 1:
        P, S = rt / top, 2.0 * ga[0] / top
        x = Ts.copy()
        for _ in range(60):
            x = x - (Q + 2.0 * k1 * (P + (S - 1.0) * x) - es * x ** 4) / (2.0 * k1 * (S - 1.0) - 4.0 * es * x ** 3)
        T0 = P + S * x
    else:
        T0 = rt / top
        x = 0.5 * (an1 + bn * T0 + T0)
    out = np.empty_like(T)
    out[0] = T0
    for i in range(1, nz):
        out[i] = (r[i] + ga[i] * out[i - 1]) / b[i]
    return {"T": np.asfortranarray(out), "Tsurf": x, "Fsurf": -(T0 - x) * cond[0] / z[0]}


def _exact_solve(c, seed):
    _, _, rowptr, col, val, E = _matrix(c, seed)
    N = E.shape[0]
    if c["method"] == "tol":
        rows = torch.from_numpy(np.repeat(np.arange(N), np.diff(rowptr)))
        cl, vl, e = torch.from_numpy(col).long(), torch.from_numpy(val), torch.from_numpy(E)
        x = e.clone()
        for _ in range(40):
            x = e + torch.zeros_like(e).index_add_(0, rows, vl * x[cl])
        return x.numpy()
    # natural row order: a forward solve, then one Gauss-Seidel sweep
    x = np.zeros(N)
    for sweep in range(2):
        old = x.copy()
        for i in range(N):
            a, b = rowptr[i], rowptr[i + 1]
            if a == b:
                x[i] = E[i]
                continue
            cc, vv = col[a:b], val[a:b]
            d = np.searchsorted(cc, i)
            x[i] = E[i] + vv[:d] @ x[cc[:d]] + (vv[d:] @ old[cc[d:]] if sweep else 0.0)
    return x


def exact(case, seed):
    if case["kind"] == "columns":
        return _exact_columns(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    return None   # ray-cast maps and step loops: a plain 64-bit program takes minutes

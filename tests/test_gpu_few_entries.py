"""Radiosity of many facets with few form factors: fewer tiles than blocks
that the passes over all facets take, in both precisions and in a batch."""
import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _ctx(ilg, level, nnz, seed=1):
    v, f = meshgen.icosphere_craters(level, 3, sigma_m=0.0, n_craters=0)
    n = f.shape[0]
    g = np.random.default_rng(seed)
    rows = np.sort(g.choice(n, nnz, replace=nnz > n))
    col = g.integers(0, n, nnz)
    key = np.unique(rows * np.int64(n) + col)
    rows, col = key // n, (key % n).astype(np.int32)
    val = g.uniform(0.1, 0.5, key.size) / np.maximum(1, np.bincount(rows, minlength=n))[rows]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    ctx = ilg.IllumContext(v, f)
    ctx.set_F(rp, col, val)
    return ctx, rows, col, val


# 3,968 facets per further block: level 4 takes 2 blocks, 5 6, 6 21
@pytest.mark.parametrize("level", [3, 4, 5, 6])
@pytest.mark.parametrize("nnz", [1, 3000, 9000, 40000])
def test_tolerance_solve(ilg, level, nnz):
    ctx, rows, col, val = _ctx(ilg, level, nnz)
    n = ctx.num_faces
    E = np.random.default_rng(2).uniform(0.0, 600.0, n)
    x, res, _ = ctx.radiosity_solve(E, tol=1e-9)
    r = np.linalg.norm(x - E - np.bincount(rows, val * x[col], n))
    assert res <= 1e-9 and r <= res + 2.0 ** -44 * np.linalg.norm(x - E) + 2.0 ** -50 * np.linalg.norm(x)
    assert np.array_equal(x[np.bincount(rows, minlength=n) == 0], E[np.bincount(rows, minlength=n) == 0])


def _model(ilg, ctx, mixed, refine):
    ctx.make_horizons(nphi=8)
    ctx.set_insolation(1, 0, 1361.0)
    dt = 6 * 3600.0 / 360
    ctx.set_suns(meshgen.spin_sun_positions(200, 6 * 3600.0, dt), ilg.fib_spiral(20))
    tm = ilg.ThermalModel(ctx, meshgen.geometric_depths(10), 300.0, 1.05e6, 220.0, emissivity=0.95,
                          bc_mode=ilg.BC_NEWTON, precision=ilg.PREC_MIXED if mixed else ilg.PREC_FP64)
    return tm, ilg.RunOpts(dt=dt, tol=1e-3 if mixed else 1e-10, max_sweeps=1 if mixed else 200, use_radiosity=1,
                           use_graph=1, precision=ilg.PREC_MIXED if mixed else ilg.PREC_FP64, coupling=1,
                           refine_every=refine)


@pytest.mark.parametrize("mixed,refine", [(0, 0), (1, 0), (1, 4)])
def test_steps_alone_and_in_a_batch(ilg, mixed, refine):
    out = []
    for batch in (False, True):
        ctxs = [_ctx(ilg, 5, nnz, seed)[0] for nnz, seed in ((200, 1), (9000, 2))]
        models = [_model(ilg, c, mixed, refine) for c in ctxs]
        if batch:
            b = ilg.Batch(ctxs, [o for _, o in models])
            b.run(12)
            b.sync()
        else:
            for c, (_, o) in zip(ctxs, models):
                c.run_steps(o, 0, 12)
        out.append([tm.T.copy() for tm, _ in models])
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("mixed,refine", [(0, 0), (1, 4)])
def test_passes_over_all_facets_take_the_device(ilg, mixed, refine):
    """One tile, 81,920 facets: 290 and 390 us by one block."""
    ctx = _ctx(ilg, 6, 100)[0]
    tm, opts = _model(ilg, ctx, mixed, refine)
    opts.use_graph = 0
    us = min(1e3 * ctx.bench_steps(opts, s, 5, flush_mb=0)[1]["radiosity"] / 5 for s in range(0, 50, 5))
    assert us < 120.0, us

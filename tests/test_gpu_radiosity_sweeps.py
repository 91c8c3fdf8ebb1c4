"""GPU parity: the FP64 tolerance solve's full and change sweeps.

The solve mixes double-float sweeps of the iterate with FP32 sweeps of its
change; whatever the mix, the returned x must satisfy the system to the
tolerance it reports, for fast and slow contractions, loose and tight
tolerances, and sweep budgets that end in either kind of sweep.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(ilg, level, albedo):
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(level, seed=5, n_craters=12, dmin_m=100.0, dmax_m=500.0)
    ctx = ilg.IllumContext(v, f)
    rp, col, val = ctx.compute_F(albedo=albedo)
    E = 600.0 * np.clip(np.cos(np.arange(f.shape[0]) * 0.37), 0.0, None)
    return ctx, rp, col, val, E


def _apply(rp, col, val, x):
    """F x, each row summed in long double."""
    p = np.concatenate([[0.0], np.cumsum((val * x[col]).astype(np.longdouble))])
    return (p[rp[1:]] - p[rp[:-1]]).astype(np.float64)


@pytest.mark.parametrize("level,albedo", [(3, 0.1), (3, 1.0), (4, 0.1), (5, 0.5)])
@pytest.mark.parametrize("tol", [1e-10, 1e-7, 1e-2])
def test_residual_within_reported_bound(ilg, level, albedo, tol):
    ctx, rp, col, val, E = _system(ilg, level, albedo)
    x, res, sweeps = ctx.radiosity_solve(E, tol=tol)
    r = np.linalg.norm(x - E - _apply(rp, col, val, x))
    # the solve's own precision: s = x - E in 48-bit sums, x in FP64
    floor = 2.0 ** -44 * np.linalg.norm(x - E) + 2.0 ** -50 * np.linalg.norm(x)
    assert 0 < sweeps <= 200 and res <= tol
    assert r <= res + floor
    xb, resb, sb = ctx.radiosity_solve(E, tol=tol)
    assert np.array_equal(x, xb) and (res, sweeps) == (resb, sb)


@pytest.mark.parametrize("budget", [1, 2, 3, 7])
def test_sweep_budget_is_jacobis(ilg, budget):
    """A budget of k sweeps ends at Jacobi's k-th iterate from x = E."""
    ctx, rp, col, val, E = _system(ilg, 4, 0.9)
    y, ys = E.copy(), []
    for _ in range(budget):
        ys.append(_apply(rp, col, val, y))
        y = E + ys[-1]
    with pytest.raises(ilg.IlgError, match=f"above tol after {budget} sweeps"):
        ctx.radiosity_solve(E, tol=1e-10, max_sweeps=budget)
    # a tolerance the k-th change meets, and no earlier one, returns the iterate itself
    d = [np.linalg.norm(b - a) for a, b in zip([np.zeros_like(E)] + ys[:-1], ys)]
    x, res, sweeps = ctx.radiosity_solve(E, tol=1.2 * d[-1], max_sweeps=budget)
    assert sweeps == budget
    # FP32 changes: 2^-23 of each change's norm, of which the first is the largest
    assert np.linalg.norm(x - y) <= 2.0 ** -23 * sum(d) + 2.0 ** -44 * np.linalg.norm(y)


@pytest.mark.parametrize("tol", [0.0, 1e-20])
def test_zero_and_tiny_tolerances_run_full_sweeps(ilg, tol):
    ctx, rp, col, val, E = _system(ilg, 3, 0.1)
    try:
        x, res, sweeps = ctx.radiosity_solve(E, tol=tol, max_sweeps=60)
    except ilg.IlgError as e:      # the iterate may cycle in its last bit
        assert "above tol after 60 sweeps" in str(e)
        return
    r = np.linalg.norm(x - E - _apply(rp, col, val, x))
    assert r <= 2.0 ** -44 * np.linalg.norm(x - E) + 2.0 ** -50 * np.linalg.norm(x)


@pytest.mark.parametrize("nnz", [1, 31, 3967, 3968, 3969, 63488, 63489, 63999, 64000, 64001, 128001])
@pytest.mark.parametrize("blocks", [0, 1, 2])
def test_tiles_of_any_entry_count(ilg, nnz, blocks):
    """Row pieces of every length (entries are stored in a bank order within
    a piece) and tiles around a group and around the largest shared tile, in
    both precisions' sweeps."""
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(3, 3, sigma_m=0.0, n_craters=0)
    n = f.shape[0]
    g = np.random.default_rng(nnz)
    lens = np.zeros(n, np.int64)
    left, i = nnz, 0
    while left > 0:   # short and long rows in turn
        k = i % n
        add = min(left, int(g.integers(1, 10)) if i % 3 else int(g.integers(1, 400)), n - 1 - int(lens[k]))
        lens[k] += add
        left -= add
        i += 1
    rp = np.concatenate([[0], np.cumsum(lens)])
    col = np.concatenate([np.sort(g.choice(n, int(m), replace=False)) for m in lens]).astype(np.int32)
    val = g.uniform(0.1, 1.0, nnz) * 0.5 / max(1, lens.max())
    ctx = ilg.IllumContext(v, f)
    ctx.set_radiosity_blocks(blocks)
    ctx.set_F(rp, col, val)
    t = ctx.F_tiles()
    assert (t["entries_per_thread"] * 992 >= 1).all() and t["rows"].sum() == (lens > 0).sum()
    if blocks:
        assert t["entries_per_thread"].max() <= max(4 * 17, -(-nnz // (992 * blocks)) + 8)
    E = g.uniform(0.0, 600.0, n)
    x, res, sweeps = ctx.radiosity_solve(E, tol=1e-9)
    r = np.linalg.norm(x - E - _apply(rp, col, val, x))
    assert res <= 1e-9 and r <= res + 2.0 ** -44 * np.linalg.norm(x - E) + 2.0 ** -50 * np.linalg.norm(x)

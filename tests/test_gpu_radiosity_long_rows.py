"""GPU parity: FP64 tolerance solves of long rows and slow contractions.

The FP32 sums of the solve's change sweeps are long here, and in the first
system they round the same way in every sweep. Whatever their errors, the
residual that the solve reports has to hold for the x it returns.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOURCES, RECEIVERS = 8000, 200


def _ctx(ilg, level, rp, col, val, blocks=0):
    from illum_gb300 import meshgen
    ctx = ilg.IllumContext(*meshgen.icosphere_craters(level, 3, sigma_m=0.0, n_craters=0))
    ctx.set_radiosity_blocks(blocks)
    ctx.set_F(rp, col, val)
    return ctx


@pytest.mark.parametrize("seed", range(6))
def test_errors_of_equal_sign_in_every_sweep(ilg, seed):
    """8,000 sources whose radiosity converges by exactly one half per sweep,
    and receivers that sum all of them with one weight: every change sweep
    adds the same numbers but for a power of two, and rounds them alike."""
    g = np.random.default_rng(seed)
    n = 20 * 4 ** 5
    e, w = g.uniform(100.0, 600.0), 50.0 * g.uniform(1.0, 2.0) / SOURCES
    col = np.concatenate([(np.arange(SOURCES) + 1) % SOURCES, np.tile(np.arange(SOURCES), RECEIVERS)]).astype(np.int32)
    val = np.concatenate([np.full(SOURCES, 0.5), np.full(SOURCES * RECEIVERS, w)])
    rp = np.full(n + 1, col.size, np.int64)
    rp[:SOURCES + 1] = np.arange(SOURCES + 1)
    rp[SOURCES:SOURCES + RECEIVERS + 1] = SOURCES + SOURCES * np.arange(RECEIVERS + 1)
    ctx = _ctx(ilg, 5, rp, col, val)
    E = np.zeros(n)
    E[:SOURCES] = e
    size = np.sqrt(RECEIVERS) * w * SOURCES * 2.0 * e      # |F x|, by far the receivers'
    for tol in size * 2.0 ** np.linspace(-19.5, -8.0, 24):
        x, res, sweeps = ctx.radiosity_solve(E, tol=tol)
        s = x[:SOURCES]
        r = np.zeros(n)
        r[:SOURCES] = s - e - 0.5 * np.roll(s, -1)
        r[SOURCES:SOURCES + RECEIVERS] = x[SOURCES:SOURCES + RECEIVERS] - w * s.astype(np.longdouble).sum()
        # double-float sums of about 700 steps (a run, then the runs of a row): (700 u)^2 of the result
        assert res <= tol and np.linalg.norm(r) <= res + 2.0 ** -29 * size, (tol, np.linalg.norm(r), res, sweeps)


def _dense(ilg, rho, blocks):
    n = 1280
    col = np.concatenate([np.delete(np.arange(n), i) for i in range(n)]).astype(np.int32)
    val = np.random.default_rng(7).uniform(0.0, 2 * rho / (n - 1), n * (n - 1))
    ctx = _ctx(ilg, 3, np.arange(n + 1, dtype=np.int64) * (n - 1), col, val, blocks)
    return ctx, col.reshape(n, -1), val.reshape(n, -1)


@pytest.mark.parametrize("rho", [0.5, 0.9, 0.97])
@pytest.mark.parametrize("blocks", [0, 26])   # the whole device, and longer runs
def test_residual_of_slow_contractions(ilg, rho, blocks):
    ctx, col, val = _dense(ilg, rho, blocks)
    E = np.random.default_rng(1).uniform(0.0, 600.0, val.shape[0])
    for tol in 10.0 ** np.linspace(-4.0, 2.0, 13):
        x, res, sweeps = ctx.radiosity_solve(E, tol=tol, max_sweeps=5000)
        r = np.linalg.norm(x - E - (val * x[col]).astype(np.longdouble).sum(1).astype(np.float64))
        # double-float sums of runs and rows of at most 170 steps: (170 u)^2 of the result
        assert res <= tol and r <= res + 2.0 ** -33 * np.linalg.norm(x), (tol, r, res, sweeps)


@pytest.mark.parametrize("rho", [0.05, 0.5, 0.9])
def test_sweep_count_is_jacobis(ilg, rho):
    """The change sweeps cost at most one sweep more than Jacobi's: the one
    that confirms a tolerance met unexpectedly."""
    ctx, col, val = _dense(ilg, rho, 0)
    E = np.random.default_rng(1).uniform(0.0, 600.0, val.shape[0])
    s, d = np.zeros_like(E), []
    for _ in range(60):
        new = (val * (E + s)[col]).sum(1)
        d.append(np.linalg.norm(new - s))
        s = new
    for tol in (1e-6, 1e-3, 1.0, 100.0):
        want = next((k + 1 for k, q in enumerate(d) if q <= tol), None)
        if want is not None:
            x, res, sweeps = ctx.radiosity_solve(E, tol=tol, max_sweeps=500)
            assert want <= sweeps <= want + 1, (tol, sweeps, want)

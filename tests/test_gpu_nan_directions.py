"""GPU: rays whose direction is not a number.

A facet with a zero normal has a finite ray origin and no direction. The
triangle test then only looks at the side a triangle lies on; a walk has to
enter every box and slab, so every ray of a closed enough mesh hits something
and each bisection goes down to its lowest end.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheet(n):
    x = (np.arange(n + 1) - n / 2) * (2.0 / n)
    X, Y = np.meshgrid(x, x, indexing="ij")
    Z = 0.05 * np.sin(9 * X) * np.cos(7 * Y) + 0.01 * np.random.default_rng(1).normal(size=X.shape)
    v = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]).ravel()
    f = np.concatenate([np.stack([i, i + n + 1, i + 1], 1), np.stack([i + 1, i + n + 1, i + n + 2], 1)])
    return v.astype(np.float32).astype(np.float64), np.ascontiguousarray(f, np.int32)


@pytest.mark.parametrize("n", [4, 8, 24])
@pytest.mark.parametrize("offset", [1e-5, 10.0])   # near and far walks
def test_horizons_without_directions(ilg, n, offset):
    v, f = _sheet(n)
    ctx = ilg.IllumContext(v, f, np.zeros((f.shape[0], 3), np.float32))
    ctx.make_horizons(nphi=9, offset=offset)
    low = np.pi / 2
    while low / 2 > 1e-3:
        low /= 2
    assert (ctx.horizons == low / 2).all()


def test_facets_without_area(ilg, oracle_mod):
    """Degenerate facets among ordinary ones: their own rays have no origin."""
    v, f = _sheet(8)
    f[5] = [3, 3, 4]
    f[40] = [10, 10, 10]
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=33)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, 33).T)

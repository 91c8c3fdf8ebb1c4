"""GPU parity: horizon and visibility rays that start far from the tree.

Large offsets along the facets' normals (also by long normals) and horizon
meshes far from the facets: the rays' origins are many times the tree's
coordinates, and the boxes they are tested against are no thicker than its
padding. Near and far rays take different walks; the line is at a quarter of
the scene's magnitude.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sheet(n=24):
    """A rough sheet of 2 n^2 facets, coordinates up to 1."""
    x = (np.arange(n + 1) - n / 2) * (2.0 / n)
    X, Y = np.meshgrid(x, x, indexing="ij")
    Z = 0.05 * np.sin(9 * X) * np.cos(7 * Y) + 0.01 * np.random.default_rng(1).normal(size=X.shape)
    v = np.stack([X.ravel(), Y.ravel(), Z.ravel()], axis=1)
    i = (np.arange(n)[:, None] * (n + 1) + np.arange(n)[None, :]).ravel()
    f = np.concatenate([np.stack([i, i + n + 1, i + 1], 1), np.stack([i + 1, i + n + 1, i + n + 2], 1)])
    return v, np.ascontiguousarray(f, np.int32)


@pytest.mark.parametrize("offset", [0.2499, 0.2501, 16.0, 300.0, 1e3, 1e4, 3e4, -0.2501, -1e4])
def test_offsets_around_and_beyond_the_line(ilg, oracle_mod, offset):
    """Bisections fine enough (1e-5) that the rays which point back at the
    sheet from far above it end at single facets."""
    v, f = _sheet()
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=9, theta_eps=1e-5, offset=offset)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, 9, theta_eps=1e-5, offset=offset).T)
    rp, col, val = ctx.compute_F(albedo=0.3, offset=offset)
    ro, co, vo, rays = oracle_mod.form_factors(v, f, albedo_scalar=0.3, offset=offset)
    rpo, cpo, vpo = oracle_mod.coo_to_csr(f.shape[0], ro, co, vo)
    assert np.array_equal(rp, rpo) and np.array_equal(col, cpo) and np.array_equal(val, vpo)
    assert ctx.visibility_rays == rays


def test_long_normals(ilg, oracle_mod):
    """The rays start at the centroid plus the offset times the given normal:
    normals of 2^14 and an offset of 1/16 are an offset of 1,024."""
    v, f = _sheet()
    v32 = v.astype(np.float32)
    n = np.cross(v32[f[:, 1]] - v32[f[:, 0]], v32[f[:, 2]] - v32[f[:, 0]]).astype(np.float64)
    n = (n / np.linalg.norm(n, axis=1)[:, None]).astype(np.float32)
    H = []
    for length, offset in ((2.0 ** 14, 2.0 ** -4), (1.0, 2.0 ** 10)):   # the same origins bit for bit
        ctx = ilg.IllumContext(v, f, n * np.float32(length))
        ctx.make_horizons(nphi=9, theta_eps=1e-5, offset=offset)
        H.append(ctx.horizons)
    assert np.array_equal(H[0], H[1])


@pytest.mark.parametrize("dist", [3.0, 100.0, 1e4, 1e5])
def test_horizon_mesh_far_from_the_facets(ilg, oracle_mod, dist):
    """Facets whose first ray points at a fine mesh far away."""
    hv, hf = _sheet(64)
    g = np.random.default_rng(2)
    tri = []
    for _ in range(256):
        u = g.normal(size=3)
        u[2] = abs(u[2]) + 0.3
        c = dist * u / np.linalg.norm(u)
        b = np.array([*g.uniform(-0.9, 0.9, 2), 0.0]) - c
        b /= np.linalg.norm(b)                      # b = t x n: the azimuth 0 at 90 degrees
        t = np.cross(b, [0.3, -0.5, 0.8])
        t /= np.linalg.norm(t)
        w = np.cross(np.cross(b, t), t)
        s = 0.02 * dist
        tri.append(np.stack([c, c + s * t, c + s * w]) - s * (t + w) / 3)
    v = np.concatenate(tri)
    f = np.arange(v.shape[0], dtype=np.int32).reshape(-1, 3)
    ctx = ilg.IllumContext(v, f)
    ctx.set_horizon_mesh(hv, hf)
    ctx.make_horizons(nphi=5)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, 5, horizon_mesh=(hv, hf)).T)

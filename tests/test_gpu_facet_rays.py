"""GPU parity: horizon and visibility rays cast by whole warps from a facet.

A warp's rays share their facet's path through the LBVH and its lanes are
refilled as rays end, so the cases that could go wrong are the ones that
leave lanes without work or put several facets into a warp: azimuth counts
around a warp's 32 lanes, and meshes around the 32-facet leaf groups.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(n_faces):
    """The first n_faces facets (Morton-coherent pieces of a cratered body)."""
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(3, seed=8, n_craters=8, dmin_m=200.0, dmax_m=600.0)
    return v, np.ascontiguousarray(f[:n_faces])


@pytest.mark.parametrize("nphi", [2, 3, 7, 8, 15, 16, 31, 32, 33, 47, 64, 65])
def test_horizons_any_azimuth_count(ilg, oracle_mod, nphi):
    v, f = _mesh(320)
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=nphi)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, nphi).T)


@pytest.mark.parametrize("n_faces", [1, 3, 5, 15, 18])
@pytest.mark.parametrize("nphi", [9, 31, 32, 63, 97, 130])
@pytest.mark.parametrize("theta_eps", [1e-3, 0.9, 4.0])   # 4: the bisection ends after one ray
def test_horizons_lanes_take_further_azimuths(ilg, oracle_mod, n_faces, nphi, theta_eps):
    v, f = _mesh(n_faces)
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=nphi, theta_eps=theta_eps)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, nphi, theta_eps=theta_eps).T)


@pytest.mark.parametrize("n_faces", [1, 2, 3, 31, 32, 33, 64, 97, 1025])
@pytest.mark.parametrize("cutoff", [None, 0.35])
def test_form_factors_around_leaf_groups(ilg, oracle_mod, n_faces, cutoff):
    v, f = _mesh(n_faces)
    ctx = ilg.IllumContext(v, f)
    rp, col, val = ctx.compute_F(albedo=0.3, cutoff=cutoff)
    ro, co, vo, rays = oracle_mod.form_factors(v, f, albedo_scalar=0.3, cutoff=-1.0 if cutoff is None else cutoff)
    rpo, cpo, vpo = oracle_mod.coo_to_csr(n_faces, ro, co, vo)
    assert np.array_equal(rp, rpo) and np.array_equal(col, cpo) and np.array_equal(val, vpo)
    assert ctx.visibility_rays == rays


@pytest.mark.parametrize("n_seen", [255, 256, 257, 511, 512, 513, 1100])
def test_form_factors_of_a_source_cast_in_parts(ilg, oracle_mod, n_seen):
    """A facet that faces n_seen others: its rays are cast in parts of 256."""
    g = np.random.default_rng(n_seen)
    u = g.normal(size=(n_seen, 3))
    u[:, 2] = np.abs(u[:, 2]) + 0.2
    c = u / np.linalg.norm(u, axis=1)[:, None] * g.uniform(0.6, 1.0, (n_seen, 1))
    tri = c[:, None, :] + 0.03 * g.normal(size=(n_seen, 3, 3))
    floor = np.array([[[0.0, 0.0, 0.0], [0.05, 0.0, 0.0], [0.0, 0.05, 0.0]]])
    v = np.concatenate([floor, tri]).reshape(-1, 3).astype(np.float32).astype(np.float64)
    f = np.arange(3 * (n_seen + 1), dtype=np.int32).reshape(-1, 3)
    ctx = ilg.IllumContext(v, f)
    rp, col, val = ctx.compute_F(albedo=0.3)
    ro, co, vo, rays = oracle_mod.form_factors(v, f, albedo_scalar=0.3, cutoff=-1.0)
    rpo, cpo, vpo = oracle_mod.coo_to_csr(n_seen + 1, ro, co, vo)
    assert np.array_equal(rp, rpo) and np.array_equal(col, cpo) and np.array_equal(val, vpo)
    assert ctx.visibility_rays == rays


@pytest.mark.parametrize("n_faces", [2047, 2048, 2049, 4097])
def test_leaf_order_around_sort_tiles(ilg, oracle_mod, n_faces):
    """The Morton keys are sorted in tiles of 2,048."""
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(4, seed=8, n_craters=8, dmin_m=200.0, dmax_m=600.0)
    f = np.ascontiguousarray(f[::-1][:n_faces])
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=2)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, 2).T)


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_horizons_of_facets_along_an_axis(ilg, oracle_mod, axis):
    """Direction components that are zero up to rounding: taken in FP64."""
    n = 9
    x, y = np.meshgrid(np.arange(n, dtype=np.float64), np.arange(n, dtype=np.float64), indexing="ij")
    z = np.zeros((n, n))
    z[4, 4] = 1.5
    v = np.roll(np.stack([x.ravel(), y.ravel(), z.ravel()], axis=1), axis, axis=1)
    i = (np.arange(n - 1)[:, None] * n + np.arange(n - 1)[None, :]).ravel()
    f = np.concatenate([np.stack([i, i + n, i + 1], axis=1), np.stack([i + 1, i + n, i + n + 1], axis=1)])
    f = np.ascontiguousarray(f, np.int32)
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=17)
    assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, 17).T)

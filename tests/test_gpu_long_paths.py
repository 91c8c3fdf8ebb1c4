"""GPU parity: facets deeper in the tree than a path has entries. The path then
ends with the whole tree in place of its upper part."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def few_entries(ilg):
    yield ilg.debug_path_entries
    ilg.debug_path_entries(0)


@pytest.mark.parametrize("entries", [1, 2, 3, 7, 13, 31])
@pytest.mark.parametrize("n_faces", [2, 3, 40, 1280])
def test_paths_that_end_with_the_whole_tree(ilg, oracle_mod, few_entries, entries, n_faces):
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(3, seed=8, n_craters=8, dmin_m=200.0, dmax_m=600.0)
    f = np.ascontiguousarray(f[:n_faces])
    few_entries(entries)
    ctx = ilg.IllumContext(v, f)
    for nphi in (9, 33):
        ctx.make_horizons(nphi=nphi)
        assert np.array_equal(ctx.horizons, oracle_mod.horizons(v, f, nphi).T)
    rp, col, val = ctx.compute_F(albedo=0.3)
    ro, co, vo, rays = oracle_mod.form_factors(v, f, albedo_scalar=0.3)
    rpo, cpo, vpo = oracle_mod.coo_to_csr(n_faces, ro, co, vo)
    assert np.array_equal(rp, rpo) and np.array_equal(col, cpo) and np.array_equal(val, vpo)
    assert ctx.visibility_rays == rays

"""The first results that a program reads: result arrays whose pages do not
exist yet take the copy no longer than a populated array and one call that
makes the pages."""
import ctypes as C
import mmap
import time

import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu

N_PHI = 4    # 0.66 MB horizon maps of 20,480 facets: 11 pages of 64 KB


@pytest.fixture(scope="module")
def ctx(ilg):
    c = ilg.IllumContext(*meshgen.icosphere_craters(5, 3, sigma_m=0.0, n_craters=0))
    c.set_horizons(np.random.default_rng(1).uniform(0.0, 1.5, (N_PHI, c.num_faces)))
    return c


def _read(ilg, ctx, fresh):
    n = 8 * ctx.num_faces * N_PHI
    m = mmap.mmap(-1, n)
    a = np.frombuffer(m, np.uint8)
    if not fresh:
        a[:] = 1
    t = time.perf_counter()
    assert ilg.lib().ilg_get_horizons(ctx._h, C.c_void_p(a.ctypes.data)) == 0
    t = time.perf_counter() - t
    assert np.array_equal(a.view(np.float64).reshape(ctx.num_faces, N_PHI).T, ctx.horizons)
    return t


def test_fresh_pages_do_not_stop_the_copy(ilg, ctx):
    _read(ilg, ctx, False)
    warm = min(_read(ilg, ctx, False) for _ in range(15))
    fresh = min(_read(ilg, ctx, True) for _ in range(15))
    # 135 us more when the copy makes the pages one by one, about 20 us in one call
    assert fresh <= warm + 8e-5, (fresh, warm)


@pytest.mark.parametrize("missing", ["first", "middle", "last", "other"])
def test_partly_fresh_arrays(ilg, ctx, missing):
    n = 8 * ctx.num_faces * N_PHI
    m = mmap.mmap(-1, n)
    a = np.frombuffer(m, np.uint8)
    q = n // 4
    for k, part in enumerate(("first", "other", "middle", "last")):
        if part != missing:
            a[k * q:(k + 1) * q] = 3
    assert ilg.lib().ilg_get_horizons(ctx._h, C.c_void_p(a.ctypes.data)) == 0
    assert np.array_equal(a.view(np.float64).reshape(ctx.num_faces, N_PHI).T, ctx.horizons)

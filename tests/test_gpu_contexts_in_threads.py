"""Contexts of different sizes set up from several threads at once: the
launch shapes of one must not change what another's launches may ask for."""
import threading

import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu

# icosphere level and azimuths: shallow and deep trees, one facet per warp and four
JOBS = [(1, 8), (5, 64), (3, 31), (5, 33), (2, 4), (4, 16)]


def test_horizons_of_several_contexts(ilg):
    ctxs = [ilg.IllumContext(*meshgen.icosphere_craters(level, 3, sigma_m=15.0, n_craters=5)) for level, _ in JOBS]
    want = []
    for c, (_, nphi) in zip(ctxs, JOBS):
        c.make_horizons(nphi=nphi)
        want.append(c.horizons)
    errors = []

    def work(c, nphi, H):
        try:
            for _ in range(400):
                c.make_horizons(nphi=nphi)
            if not np.array_equal(c.horizons, H):
                errors.append("horizons differ")
        except ilg.IlgError as e:
            errors.append(str(e))

    threads = [threading.Thread(target=work, args=(c, j[1], H)) for c, j, H in zip(ctxs, JOBS, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors

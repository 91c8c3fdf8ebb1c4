"""Results copied into fresh host arrays: the pages of the array are made
resident before the copy, in one part or several, at any alignment; bytes
beside the array stay as they are."""
import ctypes as C

import numpy as np
import pytest

import illum_gb300 as ig
from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


# horizon maps of a few bytes up to 32 MB, the smallest range whose pages are
# made resident in parts, on both sides of that line, and beyond it
@pytest.mark.parametrize("level,nphi,shift", [(1, 3, 8), (3, 13, 24), (5, 51, 8), (5, 52, 65528), (5, 204, 4096),
                                              (5, 205, 4096), (5, 301, 65528)])
def test_horizons_into_a_fresh_unaligned_array(level, nphi, shift):
    ctx = ig.IllumContext(*meshgen.icosphere_craters(level, 3, sigma_m=0.0, n_craters=0))
    n = ctx.num_faces * nphi
    H = np.random.default_rng(level * 1000 + nphi).uniform(0.0, 1.5, (nphi, ctx.num_faces))
    ctx.set_horizons(H)
    size = 8 * n + 2 * 65536
    raw = np.empty(size, np.uint8)
    start = shift + (-raw.ctypes.data) % 8
    raw[:start] = 0xA5
    raw[start + 8 * n:] = 0x5A
    rc = ig.lib().ilg_get_horizons(ctx._h, C.c_void_p(raw.ctypes.data + start))
    assert rc == 0
    got = raw[start:start + 8 * n].view(np.float64).reshape(ctx.num_faces, nphi)
    assert np.array_equal(got.T, H)
    assert (raw[:start] == 0xA5).all() and (raw[start + 8 * n:] == 0x5A).all()

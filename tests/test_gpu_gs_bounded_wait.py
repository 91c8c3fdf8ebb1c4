"""Bounded waits of the fixed-sweep Gauss-Seidel solve: a row whose columns
are not there within the poll limit ends the solve with ILG_ERR_DEVICE, and
the context stays usable. The waits run out by a limit far below the time that
a chain of dependent rows takes; no row waits for something that never comes."""
import time

import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


def test_row_wait_runs_out(ilg, oracle_mod):
    v, f = meshgen.icosphere_craters(5, 3, sigma_m=0.0, n_craters=0)
    n = f.shape[0]
    ctx = ilg.IllumContext(v, f)
    # each row depends on the one before it: a chain of 20,480 links, about a microsecond each
    rp = np.concatenate([[0, 0], np.arange(1, n)]).astype(np.int64)
    col, val = np.arange(n - 1, dtype=np.int32), np.full(n - 1, 0.5)
    ctx.set_F(rp, col, val)
    E = np.random.default_rng(1).uniform(0.0, 500.0, n)
    xo, reso, _ = oracle_mod.gauss_seidel(rp, col, val, E, mode=0, gs_steps=1)
    for polls in (1, 50):
        ctx.debug_gs_polls(polls)
        t0 = time.perf_counter()
        with pytest.raises(ilg.IlgError) as e:
            ctx.radiosity_solve_gs(E, 1)
        assert e.value.code == -6 and time.perf_counter() - t0 < 5.0       # ILG_ERR_DEVICE
    ctx.debug_gs_polls(0)
    x, res = ctx.radiosity_solve_gs(E, 1)
    assert np.array_equal(x, xo) and res == reso

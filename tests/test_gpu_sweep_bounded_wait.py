"""The wait at the end of a single mesh's FP64 sweep is bounded: with one word
that no block writes it gives up after its poll limit, the call reports
ILG_ERR_DEVICE and the context stays usable."""
import time

import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [1, 4, 8])
def test_sweep_word_wait_runs_out(ilg, oracle_mod, blocks):
    v, f = meshgen.icosphere_craters(3, seed=3, n_craters=12, dmin_m=150.0, dmax_m=450.0)
    ctx = ilg.IllumContext(v, f)
    rp, col, val = ctx.compute_F(albedo=0.1)
    t0 = time.perf_counter()
    assert ctx.debug_sweep_timeout(blocks, polls=4096, unreachable=True) == -6      # ILG_ERR_DEVICE
    assert "wait exceeded" in ilg.lib().ilg_last_error().decode()
    assert time.perf_counter() - t0 < 5.0
    assert ctx.debug_sweep_timeout(blocks, polls=4096, unreachable=False) == 0
    E = np.random.default_rng(1).uniform(0.0, 500.0, f.shape[0])
    x, res, sweeps = ctx.radiosity_solve(E, tol=1e-10, max_sweeps=200)
    xo, _, _ = oracle_mod.gauss_seidel(rp, col, val, E, mode=1, tol=1e-12, max_sweeps=500)
    assert res <= 1e-10 and np.abs(x - xo).max() <= 1e-9

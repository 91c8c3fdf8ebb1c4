"""The count of full sweeps among the FP64 solve's sweeps."""
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [0, 1])   # one tile per block, and the general kernel's first tiles
@pytest.mark.parametrize("tol,budget", [(1e-10, 200), (0.0, 5), (1e9, 200)])
def test_full_sweeps(ilg, blocks, tol, budget):
    ctx = ilg.IllumContext(*meshgen.icosphere_craters(4, seed=3, n_craters=12, dmin_m=120.0, dmax_m=400.0))
    ctx.set_radiosity_blocks(blocks)
    ctx.make_horizons(nphi=8)
    ctx.set_insolation(1, 0, 1361.0)
    ctx.compute_F(albedo=0.1, fetch=False)
    ctx.set_suns(meshgen.spin_sun_positions(20, 6 * 3600.0, 60.0), ilg.fib_spiral(20))
    tm = ilg.ThermalModel(ctx, meshgen.geometric_depths(10), 300.0, 1.05e6, 220.0, emissivity=0.95,
                          bc_mode=ilg.BC_NEWTON)
    opts = ilg.RunOpts(dt=60.0, tol=tol, max_sweeps=budget, use_radiosity=1, use_graph=1, precision=ilg.PREC_FP64,
                       coupling=1)
    ctx.bench_steps(opts, 0, 10, flush_mb=0)
    st = ctx.stats()
    if tol == 1e-10:
        assert 10 <= st["full_sweeps"] < st["radiosity_sweeps"] / 2
    else:            # every sweep of a zero tolerance, the only one of a loose one
        assert st["full_sweeps"] == st["radiosity_sweeps"] == 10 * (budget if tol == 0.0 else 1)
    ctx.set_timing(True)
    assert ctx.stats()["full_sweeps"] == 0

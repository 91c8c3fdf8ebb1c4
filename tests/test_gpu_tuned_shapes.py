"""The autotuner reports launch shapes that the steps use: mixed-precision
columns of up to 80 layers run with at most 64 threads per block, so 128 is
not among their shapes; deeper ones and FP64 columns have it."""
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz", [30, 80])
def test_mixed_columns_are_not_tuned_to_an_unused_shape(ilg, nz):
    ctx = ilg.IllumContext(*meshgen.icosphere_craters(4, seed=3, n_craters=12, dmin_m=120.0, dmax_m=400.0))
    ctx.make_horizons(nphi=16)
    ctx.set_insolation(1, 0, 1361.0)
    ctx.compute_F(albedo=0.1, fetch=False)
    ctx.set_suns(meshgen.spin_sun_positions(2, 6 * 3600.0, 60.0), ilg.fib_spiral(100))
    tm = ilg.ThermalModel(ctx, meshgen.geometric_depths(nz), 300.0, 1.05e6, 220.0, emissivity=0.95,
                          bc_mode=ilg.BC_NEWTON, precision=ilg.PREC_MIXED)
    opts = ilg.RunOpts(dt=60.0, tol=1e-3, max_sweeps=1, use_radiosity=1, use_graph=1, precision=ilg.PREC_MIXED,
                       coupling=1)
    # (with 128 timed as one more run of the 64-thread launch, it would win a good part of the time)
    for _ in range(20):
        assert ctx.autotune(opts)["conduct_threads"] in (32, 64)
    ctx.set_tune(256, 8, 128)      # accepted as before
    ctx.run_steps(opts, 0, 1)

"""The count of facets that the direct insolation leaves to the exact test,
as ilg_get_stats adds it up over steps: captured steps, whose insolation of a
later frame runs in a kernel of its own beside the radiosity solve, count what
serial steps count for the same frame."""
import numpy as np
import pytest

from illum_gb300 import meshgen

pytestmark = pytest.mark.gpu


# levels 5 and 6: more facets than one turn of the 152 blocks takes
@pytest.mark.parametrize("level,mixed,refine", [(3, 0, 0), (5, 0, 0), (5, 1, 0), (5, 1, 3), (6, 1, 3)])
def test_count_per_frame(ilg, level, mixed, refine):
    v, f = meshgen.icosphere_craters(level, seed=3, n_craters=12, dmin_m=120.0, dmax_m=400.0)
    ctx = ilg.IllumContext(v, f)
    ctx.make_horizons(nphi=16)
    ctx.set_insolation(1, 0, 1361.0)
    ctx.compute_F(albedo=0.1, fetch=False)
    dt, n = 6 * 3600.0 / 90, 14
    ctx.set_suns(meshgen.spin_sun_positions(n, 6 * 3600.0, dt), ilg.fib_spiral(100))
    tm = ilg.ThermalModel(ctx, meshgen.geometric_depths(10), 300.0, 1.05e6, 220.0, emissivity=0.95,
                          bc_mode=ilg.BC_NEWTON, precision=ilg.PREC_MIXED if mixed else ilg.PREC_FP64)

    def counts(graph):
        opts = ilg.RunOpts(dt=dt, tol=1e-3 if mixed else 1e-10, max_sweeps=1 if mixed else 200, use_radiosity=1,
                           use_graph=graph, precision=ilg.PREC_MIXED if mixed else ilg.PREC_FP64, coupling=1,
                           refine_every=refine)
        got = [ctx.stats()["ambiguous_facets"]]
        for s in range(n - 3):
            ctx.bench_steps(opts, s, 1, flush_mb=0)
            got.append(ctx.stats()["ambiguous_facets"])
        return np.diff(got)

    serial, graph = counts(0), counts(1)
    assert serial.max() > 0 and len(set(serial.tolist())) > 1
    # a captured step looks one frame further ahead than a serial one
    assert np.array_equal(graph[:-1], serial[1:])

"""GPU: kernels of a time step at the edges of their chunks and blocks.

Conduction: columns pass eight layers at a time, FP32 columns live in
registers in classes of 32, 48, 64 and 80 layers, deeper ones in shared
memory. Direct insolation beside the radiosity solve: blocks of 128 or 256
facets and a list of the pairs they test exactly; the serial order uses other
kernels, and both must agree bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _piece(n_faces, level=3):
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(level, seed=8, n_craters=8, dmin_m=200.0, dmax_m=600.0)
    return v, np.ascontiguousarray(f[:n_faces])


@pytest.mark.parametrize("nz", [2, 3, 7, 8, 9, 10, 16, 17, 18, 31, 32, 33, 47, 48, 49, 63, 64, 65, 79, 80, 81])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_columns_of_any_depth_vs_oracle(ilg, oracle_mod, nz, precision):
    v, f = _piece(70)
    n = f.shape[0]
    g = np.random.default_rng(nz)
    z = 0.5 * np.arange(1, nz + 1) / nz          # equal layers: a step amplifies no rounding
    ti, rhoc = np.full(nz, 300.0), np.full(nz, 1.05e6)
    T = np.empty((nz + 1, n))
    T[0] = g.uniform(150.0, 300.0, n)
    T[1:] = 220.0 + (T[0] - 220.0) * np.exp(-z / 0.1)[:, None] + g.normal(0.0, 2.0, (nz, n))
    ctx = ilg.IllumContext(v, f)
    tm = ilg.ThermalModel(ctx, z, 300.0, 1.05e6, T,
                          precision=ilg.PREC_MIXED if precision == "mixed" else ilg.PREC_FP64)
    Q = g.uniform(0.0, 700.0, n)
    tm.step(60.0, Q)
    out = np.empty_like(T)
    for k in range(n):
        out[1:, k], out[0, k], _ = oracle_mod.conductionq(z, 60.0, 0.0, Q[k], T[1:, k], ti, rhoc, 0.999, T[0, k])
    if precision == "fp64":
        tol = 1e-9
    else:   # T rounded to FP32 before and after, and the increments' own rounding
        tol = (2.0 * np.sqrt(nz) + 2.0) * 2.0 ** -24 * T.max() + 2.0 ** -18 * np.abs(out - T).max()
    assert np.abs(tm.T - out).max() <= tol


@pytest.mark.parametrize("n_faces,ndisk", [(1, 100), (127, 100), (128, 2), (129, 100), (255, 37), (256, 100),
                                           (257, 100), (640, 700), (1280, 700)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("norm_mode,interp", [(0, 0), (1, 1)])
def test_insolation_beside_the_solve_equals_serial_order(ilg, n_faces, ndisk, precision, norm_mode, interp):
    from illum_gb300 import meshgen
    v, f = _piece(n_faces)
    prec = ilg.PREC_MIXED if precision == "mixed" else ilg.PREC_FP64
    got = []
    for serial in (False, True):
        ctx = ilg.IllumContext(v, f)
        ctx.make_horizons(nphi=32)
        ctx.set_insolation(norm_mode, interp, 1361.0)
        ctx.compute_F(albedo=0.1, fetch=False)
        ctx.set_suns(meshgen.spin_sun_positions(12, 6 * 3600.0, 1800.0), ilg.fib_spiral(ndisk))
        tm = ilg.ThermalModel(ctx, meshgen.geometric_depths(30), 200.0, 1.05e6, 200.0, emissivity=0.95,
                              bc_mode=ilg.BC_NEWTON, precision=prec)
        if prec == ilg.PREC_MIXED:
            o = ilg.RunOpts(dt=1800.0, tol=1e-3, max_sweeps=1, use_radiosity=1, use_graph=1, precision=prec,
                            coupling=ilg.COUPLE_DIRECT, refine_every=4)
        else:
            o = ilg.RunOpts(dt=1800.0, tol=1e-10, max_sweeps=200, use_radiosity=1, use_graph=1, precision=prec,
                            coupling=ilg.COUPLE_DIRECT)
        ctx.set_timing(serial)     # phase-timed steps run in the serial order
        ts = ctx.run_steps(o, 0, 12, record_tsurf=True)
        got.append((ts, ctx.outputs()["rad"], tm.T))
    for a, b in zip(*got):
        assert np.array_equal(a, b)

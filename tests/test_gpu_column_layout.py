"""GPU: standalone batched columns at the edges of their layout tiles.

Columns change between the caller's layout and the device's in 32 x 32 tiles
and run 32 per block. A column's arithmetic does not depend on the columns
beside it, so a batch must equal its columns one at a time bit for bit, for
counts of columns and layers around those sizes and for columns too deep for
shared memory (single columns against the oracle: test_gpu_parity).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncol", [2, 31, 32, 33, 65])
@pytest.mark.parametrize("nz", [2, 31, 32, 33, 64, 161, 700])
@pytest.mark.parametrize("bc", [0, 1])
def test_batch_equals_single_columns(ilg, ncol, nz, bc):
    g = np.random.default_rng(1000 * nz + ncol)
    z = 0.5 * np.arange(1, nz + 1) / nz
    T = 200.0 + 30.0 * g.normal(size=(nz, ncol))
    Ts = 210.0 + 30.0 * g.normal(size=ncol)
    Qn, Q = g.uniform(0.0, 600.0, (2, ncol))
    ti, rhoc = np.full(nz, 300.0), np.full(nz, 1.05e6)
    Tg, Tsg, Fg = ilg.conductionQ_batch(z, 60.0, Qn, Q, T, ti, rhoc, 0.95, Ts, 0.02, bc_mode=bc)
    for f in range(ncol):
        T1, Ts1, F1 = ilg.conductionQ_batch(z, 60.0, Qn[f:f + 1], Q[f:f + 1], T[:, f:f + 1], ti, rhoc, 0.95,
                                            Ts[f:f + 1], 0.02, bc_mode=bc)
        assert np.array_equal(Tg[:, f], T1[:, 0]) and Tsg[f] == Ts1[0] and Fg[f] == F1[0]

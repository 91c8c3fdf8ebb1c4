"""ilg_set_radiosity_blocks cuts the row tiles for the block count that the
caller asks for, also where that makes them large."""
import numpy as np
import pytest

import illum_gb300 as ig


def test_blocks_for_a_mesh():
    assert ig.radiosity_blocks_for(1_000_000, 200_000) == 5
    assert ig.radiosity_blocks_for(1_000_001, 200_000) == 6
    assert ig.radiosity_blocks_for(0) == ig.radiosity_blocks_for(1) == ig.radiosity_blocks_for(20_000) == 1
    assert ig.radiosity_blocks_for(20_001) == 2
    assert ig.radiosity_blocks_for(480_000) == 24 and ig.radiosity_blocks_for(1_000_000) == 25
    assert ig.radiosity_blocks_for(64_000 * 100) == 100


@pytest.mark.gpu
@pytest.mark.parametrize("blocks", [1, 2, 5, 12])
def test_tiles_follow_the_block_count(ilg, blocks):
    from illum_gb300 import meshgen
    v, f = meshgen.icosphere_craters(3, 3, sigma_m=0.0, n_craters=0)
    n, m = f.shape[0], 500
    g = np.random.default_rng(1)
    col = np.concatenate([np.sort(g.choice(n, m, replace=False)) for _ in range(n)]).astype(np.int32)
    val = g.uniform(0.0, 1.0 / m, n * m)
    ctx = ilg.IllumContext(v, f)
    ctx.set_F(np.arange(n + 1, dtype=np.int64) * m, col, val)
    ctx.set_radiosity_blocks(blocks)
    t = ctx.F_tiles()
    # equal shares, but tiles above twice 131,072 entries are halved
    assert blocks <= len(t["rows"]) <= max(blocks, 2 * -(-n * m // 262_144)), t
    E = g.uniform(0.0, 600.0, n)
    x, res, _ = ctx.radiosity_solve(E, tol=1e-8)
    r = np.linalg.norm(x - E - (val * x[col]).reshape(n, m).astype(np.longdouble).sum(1).astype(np.float64))
    assert res <= 1e-8 and r <= res + 2.0 ** -36 * np.linalg.norm(x)

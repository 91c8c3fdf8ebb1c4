"""The set-up's radix sort against numpy's stable sort: around the tiles of
both tile sizes and the line between them, with and without values, and with
tiles that give up looking for the counts of the tiles before them and count
the keys themselves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMALL, LARGE, LINE = 2048, 6144, 1 << 19


def _check(ilg, n, bits, polls, values, seed):
    g = np.random.default_rng(seed)
    keys = g.integers(0, 1 << 62, n, dtype=np.uint64) * np.uint64(4) + g.integers(0, 4, n, dtype=np.uint64)
    keys >>= np.uint64(64 - bits)
    keys[g.random(n) < 0.3] = keys[0]                      # many equal keys: the order of their values shows
    if bits >= 16:
        keys[g.random(n) < 0.2] &= np.uint64(0xff)         # and many that share their high digits
    order = np.argsort(keys, kind="stable")
    if values:
        k, v = ilg.debug_sort(keys, np.arange(n), bits, polls)
        assert np.array_equal(v, order)
    else:
        k = ilg.debug_sort(keys, None, bits, polls)
    assert np.array_equal(k, keys[order])


@pytest.mark.parametrize("n", [1, 2, 31, SMALL - 1, SMALL, SMALL + 1, 9 * SMALL + 1, LINE - 1, LINE, LINE + 1,
                               86 * LARGE - 1, 86 * LARGE, 86 * LARGE + 1, 163 * LARGE + 7])
@pytest.mark.parametrize("values", [False, True])
@pytest.mark.parametrize("polls", [-1, 0])
def test_sizes(ilg, n, values, polls):
    _check(ilg, n, 34, polls, values, n)


@pytest.mark.parametrize("bits", [1, 7, 8, 9, 16, 17, 40, 63, 64])
@pytest.mark.parametrize("n", [5 * SMALL + 3, LINE + LARGE // 2])
@pytest.mark.parametrize("polls", [-1, 0, 1])
def test_key_widths(ilg, bits, n, polls):
    _check(ilg, n, bits, polls, True, bits)

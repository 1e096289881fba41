"""GPU tests of the preprocessing sort (csrc/primitives.cuh) at the sizes where
its tiles and passes change: the oriented CSR equals the oracle's in every
offset and column."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FEW, FULL, LINE = 1536, 6144, 148 * 1536  # tiles for few keys, many; the line between


@pytest.mark.parametrize("pairs", [1, 31, FEW - 1, FEW, FEW + 1, FULL, FULL + 1, 20 * FEW + 5,
                                   LINE - 1, LINE, LINE + 1, 500_003])
@pytest.mark.parametrize("n", [2, 120, 3000, 65_537])
def test_orientation_at_tile_edges(wetric_mod, oracle_mod, pairs, n):
    """n sets the digits: 2 to 34 key bits (1 to 5 passes of 7 or 8 bits, in the low and
    the high word); small n means runs of duplicates and loops."""
    rng = np.random.default_rng(pairs * 7 + n)
    src = rng.integers(0, n, pairs).astype(np.uint32)
    dst = np.minimum((n * rng.random(pairs) ** 3).astype(np.uint32), n - 1)  # skewed
    want = oracle_mod.oriented_from_pairs(src, dst, n)
    g = wetric_mod.orient_edges(src, dst, n=n)
    got = g.download()
    g.free()
    assert np.array_equal(got.row_ptr, want.row_ptr)
    assert np.array_equal(got.col_ind, want.col_ind)

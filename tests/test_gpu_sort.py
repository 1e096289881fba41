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


@pytest.mark.parametrize("size", [2, 5, 32, 33, 34, 130, 512, 513, 514, 600])
def test_symmetric_rows_around_the_row_sort(wetric_mod, oracle_mod, size):
    """A clique of `size` gives an oriented row of size - 1 columns: around a
    warp's and the in-place rows' 512, where the radix sort takes over; with
    a sparse graph, hubs and isolated vertices beside it, host and device."""
    import torch

    rng = np.random.default_rng(size)
    n = 4000
    i, j = np.triu_indices(size, 1)
    ids = rng.permutation(n - 500)  # the last 500 stay isolated
    src = np.concatenate([ids[i], rng.integers(0, n - 500, 9000), np.full(900, ids[700])])
    dst = np.concatenate([ids[j], rng.integers(0, n - 500, 9000), ids[1000:1900]])
    sym = oracle_mod.csr_from_pairs(src.astype(np.uint32), dst.astype(np.uint32), n)
    want = oracle_mod.preprocess(sym)
    got = wetric_mod.preprocess(wetric_mod.Graph(sym.row_ptr, sym.col_ind))
    assert np.array_equal(got.row_ptr, want.row_ptr)
    assert np.array_equal(got.col_ind, want.col_ind)
    tri = oracle_mod.count_merge(want)
    rp = torch.from_numpy(sym.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(sym.col_ind.view(np.int32)).cuda()
    assert wetric_mod.count(rp, ci, 5, 64, oriented=False)[0] == tri
    assert wetric_mod.count(rp.int(), ci, 5, 64, oriented=False)[0] == tri


@pytest.mark.parametrize("hubs", [1, 2, 7])
@pytest.mark.parametrize("leaves", [1, 30, 126, 127, 128, 129, 161, 5000])
def test_symmetric_hubs_in_place(wetric_mod, oracle_mod, hubs, leaves):
    """Rows of hubs that keep nothing or little of many columns, around the
    128 columns from which such rows are skipped."""
    rng = np.random.default_rng(hubs * 7 + leaves)
    n = hubs + leaves + 40
    ids = rng.permutation(n)
    i, j = np.triu_indices(hubs, 1)
    src = np.concatenate([np.repeat(np.arange(hubs), leaves), i, hubs + rng.integers(0, leaves, 20)])
    dst = np.concatenate([np.tile(hubs + np.arange(leaves), hubs), j,
                          hubs + rng.integers(0, leaves, 20)])
    sym = oracle_mod.csr_from_pairs(ids[src].astype(np.uint32), ids[dst].astype(np.uint32), n)
    want = oracle_mod.preprocess(sym)
    got = wetric_mod.preprocess(wetric_mod.Graph(sym.row_ptr, sym.col_ind))
    assert np.array_equal(got.row_ptr, want.row_ptr)
    assert np.array_equal(got.col_ind, want.col_ind)

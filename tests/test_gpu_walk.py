"""GPU tests of the column walk (csrc/walk.cuh): the wedges below the core
counted by middle vertex, at the sizes where its pieces change -- rows past
one hash set's columns, vertices past one piece of entries, light vertices at
their limits, no core and cores of several lengths, wedge ranges that cut
rows and tails, and host input in row chunks. Counts are exact: every one
equals the oracle's.
"""
import numpy as np
import pytest

from conftest import complete_graph, comb3

pytestmark = pytest.mark.gpu


def graph(oracle_mod, kind):
    rng = np.random.default_rng(77)
    if kind == "rmat":
        import wetric

        src, dst = wetric.gen_rmat(16, 16 << 16, seed=5)
    elif kind == "dense":  # rows of 700 to 2,600 columns: several set sizes, two parts
        n = 3000
        i, j = np.triu_indices(n, 1)
        keep = rng.random(i.size) < np.where(i < 400, 0.97, 0.45)
        src, dst = i[keep], j[keep]
    elif kind == "hub":  # short rows all ending in a few hubs: many pieces per w
        m = 120_000
        leaf = np.repeat(np.arange(m), 32)
        src, dst = leaf, m + rng.integers(0, 90, leaf.size)
        i, j = np.triu_indices(90, 1)
        src, dst = np.concatenate([src, m + i]), np.concatenate([dst, m + j])
    else:  # "light": d+ around 64 and entries around 128
        n = 20_000
        src = rng.integers(0, n, 64 * n)
        dst = (src + rng.integers(1, 130, src.size)) % n
    return oracle_mod.oriented_from_pairs(src.astype(np.uint32), dst.astype(np.uint32))


@pytest.mark.parametrize("kind", ["rmat", "dense", "hub", "light"])
def test_walk_parity(wetric_mod, oracle_mod, kind):
    import torch

    g = graph(oracle_mod, kind)
    want = oracle_mod.count_merge(g)
    W = oracle_mod.wedge_total(g)
    assert W >= 4 * g.m + (16 << 20), (W, g.m)  # enough wedges for the walk
    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    rp32 = rp.int()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    for core in (wetric_mod.CORE_OFF, 0, 32, 1000):
        for kw in ({}, {"pair_streams": False}, {"one_pass": True}, {"validate": True},
                   {"keep_u64_offsets": True}, {"kernel": 8}):
            got, st = wetric_mod.count(rp, ci, 5, 8192, core_len=core, **kw)
            assert got == want, (kind, core, kw)
            assert st.wedges == W and st.wedges_counted == W
        assert wetric_mod.count(rp32, ci, 1, 0, core_len=core)[0] == want


@pytest.mark.parametrize("kind", ["rmat", "dense"])
def test_walk_wedge_ranges(wetric_mod, oracle_mod, kind):
    """Ranges large enough to walk, their ends inside rows and tails."""
    g = graph(oracle_mod, kind)
    W = oracle_mod.wedge_total(g)
    rng = np.random.default_rng(3)
    need = 4 * g.m + (16 << 20)
    for core in (wetric_mod.CORE_OFF, 500):
        for _ in range(4):
            b = int(rng.integers(0, W - need))
            e = int(rng.integers(b + need, W + 1))
            got, st = wetric_mod.count(g.row_ptr, g.col_ind, 5, 8192, wedge_begin=b,
                                       wedge_end=e, core_len=core)
            rest = [wetric_mod.count(g.row_ptr, g.col_ind, 5, 8192, wedge_begin=x, wedge_end=y,
                                     core_len=core, kernel=8)[0]
                    for x, y in ((b, b + 7), (b + 7, e - 5), (e - 5, e))]
            assert st.wedges_counted == e - b
            assert got == sum(rest), (core, b, e)


def test_walk_host_row_chunks(wetric_mod, oracle_mod):
    src, dst = wetric_mod.gen_rmat(19, 16 << 19, seed=21)
    g = oracle_mod.oriented_from_pairs(src, dst)
    assert g.m >= 1 << 22
    want = oracle_mod.count_merge(g)
    for core in (wetric_mod.CORE_OFF, 0, 4096):
        assert wetric_mod.count(g.row_ptr, g.col_ind, 5, 8192, core_len=core)[0] == want


def test_walk_on_a_clique(wetric_mod, oracle_mod):
    """Rows of up to 2,199 columns, every wedge closed: hash sets in two
    parts (no core) and the whole graph in the core."""
    k = 2200
    g = oracle_mod.oriented_from_pairs(*complete_graph(k))
    for core in (wetric_mod.CORE_OFF, 40, 0):
        assert wetric_mod.count(g.row_ptr, g.col_ind, 5, 64, core_len=core)[0] == comb3(k)


def test_walk_without_room_falls_back(wetric_mod, oracle_mod):
    """Under a budget that has no room for the walk's entries the count takes
    the wedge-check path and is the same."""
    import torch

    g = graph(oracle_mod, "rmat")
    want = oracle_mod.count_merge(g)
    rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    try:
        wetric_mod.set_hbm_budget(12 << 20)
        assert wetric_mod.count(rp, ci, 5, 0, core_len=wetric_mod.CORE_OFF)[0] == want
    finally:
        wetric_mod.set_hbm_budget(0)


def test_small_graphs_in_one_pass(wetric_mod, oracle_mod):
    """Graphs below the size of a core and a walk, with rows longer than a
    short row, at the edges of the tiles, u64 and u32 offsets, columns at
    every alignment, and offsets that do not fit them."""
    import torch

    rng = np.random.default_rng(8)
    for n, pairs in ((2, 1), (3, 3), (40, 700), (33, 31), (300, 4000), (700, 100000),
                     (5000, 20001)):
        src, dst = (rng.integers(0, n, pairs).astype(np.uint32) for _ in range(2))
        g = oracle_mod.oriented_from_pairs(src, dst)
        want, W = oracle_mod.count_merge(g), oracle_mod.wedge_total(g)
        d = np.diff(g.row_ptr.astype(np.int64))
        for off in range(8 if n == 300 else 2):
            ci = torch.zeros(g.m + off, dtype=torch.int32, device="cuda")[off:]
            ci.copy_(torch.from_numpy(g.col_ind.view(np.int32)))
            for dt in (np.int32, np.int64):
                rp = torch.from_numpy(g.row_ptr.astype(dt)).cuda()
                got, st = wetric_mod.count(rp, ci, 5, 8192)
                assert (got, st.wedges) == (want, W)
                assert st.max_out_degree == (d.max() if d.size else 0)
                if g.m > 2:
                    bad = rp.clone()
                    bad[1] = g.m + 5
                    with pytest.raises(wetric_mod.WetricError):
                        wetric_mod.count(bad, ci, 5, 8192)


@pytest.mark.parametrize("use_graph", [False, True])
def test_batch_walk(wetric_mod, oracle_mod, use_graph):
    """A batch whose long rows are walked per graph: graphs past one
    65,536-bit window beside tiny and empty ones, so that graph boundaries
    fall inside windows, tiles and groups of entries; every count repeated."""
    rng = np.random.default_rng(3)
    parts, n = [], []
    for kind in ("rmat", "dense", "hub"):
        g = graph(oracle_mod, kind)
        i = np.repeat(np.arange(g.n), np.diff(g.row_ptr.astype(np.int64)))
        parts.append((i.astype(np.uint32), g.col_ind.astype(np.uint32)))
        n.append(g.n)
        for size in (1, 3, 40, 700):
            e = 0 if size == 1 else 6 * size
            parts.append(tuple(rng.integers(0, size, e).astype(np.uint32) for _ in "sd"))
            n.append(size)
    order = rng.permutation(len(parts))
    parts, n = [parts[i] for i in order], [n[i] for i in order]
    want = [oracle_mod.count_merge(oracle_mod.oriented_from_pairs(*p)) if p[0].size else 0
            for p in parts]
    src, dst = (np.concatenate([p[k] for p in parts]) for k in (0, 1))
    off = np.concatenate([[0], np.cumsum([p[0].size for p in parts])]).astype(np.uint64)
    args = (src, dst, off, np.array(n, np.uint64))
    b = wetric_mod.Batch(*args, use_cuda_graph=use_graph)
    for _ in range(3):
        got, _ = b.count()
        assert [int(x) for x in got] == want
    got, _ = wetric_mod.Batch(*args, use_cuda_graph=use_graph, pair_streams=False).count()
    assert [int(x) for x in got] == want


@pytest.mark.parametrize("degree", [17, 20, 31, 33, 48, 49, 63, 66])
@pytest.mark.parametrize("window", [70, 4000])
def test_row_sets_parity(wetric_mod, oracle_mod, degree, window):
    """Rows around one warp, a set's 64 columns and the short rows' 48: enough
    edges per row for the sets, columns close together (`window`: neighbours
    among the next ids, so shared columns and triangles are many) and spread."""
    rng = np.random.default_rng(degree * 31 + window)
    n = 2_000_000 // degree
    src = np.repeat(np.arange(n), degree)
    dst = (src + 1 + rng.integers(0, window, src.size)) % n
    g = oracle_mod.oriented_from_pairs(src.astype(np.uint32), dst.astype(np.uint32))
    want = oracle_mod.count_merge(g)
    W = oracle_mod.wedge_total(g)
    assert g.m >= 1 << 20 and W >= 8 * g.m  # enough for the sets
    import torch

    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    for core in (wetric_mod.CORE_OFF, 0):
        got, st = wetric_mod.count(rp, ci, 5, 8192, core_len=core)
        assert got == want and st.wedges == W and st.wedges_counted == W
    # the same columns at an odd place in their sector
    ci1 = torch.cat([ci[:3], ci])[3:]
    assert wetric_mod.count(rp, ci1, 5, 8192)[0] == want
    # twice in a batch, with a small graph between
    off = np.array([0, src.size, src.size + 3, 2 * src.size + 3], np.uint64)
    s = np.concatenate([src, [0, 1, 2], src]).astype(np.uint32)
    d = np.concatenate([dst, [1, 2, 0], dst]).astype(np.uint32)
    counts, _ = wetric_mod.Batch(s, d, off, np.array([n, 3, n], np.uint64)).count()
    assert [int(x) for x in counts] == [want, 1, want]


@pytest.mark.parametrize("n,edges", [(2, 1), (33, 400), (70, 2000), (9000, 131_000),
                                     (60_000, 131_071), (60_000, 131_072), (1 << 20, 60_000),
                                     ((1 << 20) + 1, 60_000)])
def test_small_graph_parity(wetric_mod, oracle_mod, n, edges):
    """Around the single launch's limits: its columns (2^17), its rows (2^20),
    fewer edges than a warp, long runs of empty rows, a row of every edge."""
    import torch

    rng = np.random.default_rng(n + edges)
    for hub in (False, True):
        if hub:  # one row past several warps' edges
            k = min(n - 1, edges)
            src = np.zeros(k, np.int64)
            dst = 1 + np.arange(k)
            extra = rng.integers(0, n, (2, max(0, edges - k)))
            src, dst = np.concatenate([src, extra[0]]), np.concatenate([dst, extra[1]])
            key = np.unique(np.minimum(src, dst) * n + np.maximum(src, dst))
        else:
            pair = rng.integers(0, n, (2, 2 * edges + 20)) if n > 2 else np.array([[0], [1]])
            key = np.unique(pair.min(0) * n + pair.max(0))
            key = rng.permutation(key[key // n != key % n])[:edges]
        key = np.sort(key[key // n != key % n])
        rp = np.zeros(n + 1, np.uint64)  # an oriented CSR in id order
        rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
        ci = (key % n).astype(np.uint32)
        g = oracle_mod.CSR(rp, ci)
        want, W = oracle_mod.count_merge(g), oracle_mod.wedge_total(g)
        rp64 = torch.from_numpy(rp.view(np.int64)).cuda()
        col = torch.from_numpy(ci.view(np.int32)).cuda()
        odd = torch.cat([col[:1], col])[1:]
        for r, c in ((rp64, col), (rp64.int(), col), (rp64.int(), odd)):
            for kw in ({}, {"validate": True}):
                got, st = wetric_mod.count(r, c, 5, 8192, **kw)
                assert got == want and st.wedges == st.wedges_counted == W
                assert st.max_out_degree == int(np.diff(rp.astype(np.int64)).max())

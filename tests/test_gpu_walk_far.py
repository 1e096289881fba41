"""GPU tests of the walk's columns outside the window (csrc/walk.cuh): long rows
with more than 48 columns below the last 65,536 vertices, so that tails split
into a window entry and a rest entry, rest sets are hash sets of one and of
several parts, for blocks and for single warps, and entries outgrow their
room. The graphs are CSRs in id order; what each one reaches is worked out
from its rows first.
"""
import numpy as np
import pytest

from conftest import comb3

pytestmark = pytest.mark.gpu
WINDOW, SHORT, PART, FEW = 65_536, 48, 1024, 64


def csr(oracle_mod, n, src, dst):
    key = np.unique(src.astype(np.int64) * n + dst)
    rp = np.zeros(n + 1, np.uint64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return oracle_mod.CSR(rp, (key % n).astype(np.uint32))


def far_graph(oracle_mod, kind):
    """Vertices of the dense part lie below the window, in between empty rows."""
    rng = np.random.default_rng(11)
    n = 270_000
    share = 0.2  # of the vertices have window columns (all: no room for the entries)
    if kind in ("parts", "heavy"):  # rows of up to 1,150 or 1,800 columns outside the window
        k, p, win = 3000, 0.35 if kind == "parts" else 0.6, 60
        i, j = np.triu_indices(k, 1)
        keep = rng.random(i.size) < p
        i, j = i[keep], j[keep]
    elif kind == "light":  # rows and entries of around 64
        k, win = 20_000, 6
        i = np.repeat(np.arange(k), 74)
        j = i + rng.integers(1, 300, i.size)
        i, j = i[j < k], j[j < k]
    else:  # "hub": nearly all rows end in 30 long ones: many pieces of entries
        k, win, share = 60_000, 3, 1.0
        i = np.repeat(np.arange(k - 400), 12)
        j = k - 400 + rng.integers(0, 30, i.size)
        a, b = np.triu_indices(400, 1)
        i, j = np.concatenate([i, k - 400 + a]), np.concatenate([j, k - 400 + b])
    at = np.sort(rng.choice(n - WINDOW - 10, k, replace=False))
    to = np.repeat(at[rng.random(k) < share], win)
    to = to, n - 1 - rng.integers(0, WINDOW, to.size)
    near = np.sort(n - 1 - rng.integers(0, WINDOW, (300_000, 2)), axis=1)
    near = near[near[:, 0] < near[:, 1]]
    return csr(oracle_mod, n, np.concatenate([at[i], to[0], near[:, 0]]),
               np.concatenate([at[j], to[1], near[:, 1]]))


def entries(g):
    """(rest entries per middle vertex, window entries, rest columns of its row)."""
    n = g.n
    rp, ci = g.row_ptr.astype(np.int64), g.col_ind.astype(np.int64)
    d = np.diff(rp)
    row = np.repeat(np.arange(n), d)
    far = np.bincount(row, weights=ci < n - WINDOW, minlength=n).astype(np.int64)
    cut = rp[:-1] + far
    long = d > SHORT
    j = np.arange(ci.size)
    to_long = long[ci]
    rest = to_long & (j + 1 < cut[row]) & (far[ci] > SHORT)
    win = to_long & (np.maximum(j + 1, cut[row]) < rp[1:][row])
    return np.bincount(ci[rest], minlength=n), int(win.sum()), far


KINDS = ["parts", "light", "hub"]


def heavy(g, far):
    """Bound of the wedges outside the window between rows that take several
    hash sets there."""
    far = far[far > PART]
    return min(int((far * (far - 1) // 2).sum()), int(far.sum()) * far.size)


@pytest.mark.parametrize("kind", KINDS)
def test_far_columns(wetric_mod, oracle_mod, kind):
    import torch

    g = far_graph(oracle_mod, kind)
    rest, win, far = entries(g)
    d = np.diff(g.row_ptr.astype(np.int64))
    assert rest.sum() > 10_000 and win > 10_000
    assert rest.sum() + win < g.m + g.m // 4  # they have room
    assert g.m >= 1 << 19 and (d.max() > 128 or (d * (d - 1) // 2)[d > SHORT].sum() >= 1 << 25)
    assert heavy(g, far) <= oracle_mod.wedge_total(g) // 10
    one_warp = (rest > 0) & (rest <= FEW) & (far <= 128)
    if kind == "parts":
        assert (far[rest > 0] > PART).sum() > 30  # sets in two parts
    elif kind == "light":
        assert one_warp.sum() > 1000 and ((rest > 0) & ~one_warp).sum() > 1000
    else:
        assert rest.max() > 2 * 2048  # pieces
    want, W = oracle_mod.count_merge(g), oracle_mod.wedge_total(g)
    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    for core in (wetric_mod.CORE_OFF, 0, 32, 1000, 40_000, 65_536):
        for kw in ({}, {"one_pass": True}, {"validate": True}, {"kernel": 8}):
            got, st = wetric_mod.count(rp, ci, 5, 8192, core_len=core, **kw)
            assert got == want and st.wedges == st.wedges_counted == W, (core, kw)
            if "kernel" not in kw:
                assert st.pair_wedges + st.core_wedges < W  # the rest were walked
    for off in range(1, 8):  # columns at every place in their sector
        c = torch.zeros(g.m + off, dtype=torch.int32, device="cuda")[off:]
        c.copy_(ci)
        assert wetric_mod.count(rp.int(), c, 5, 8192)[0] == want
    assert wetric_mod.count(g.row_ptr, g.col_ind, 5, 8192)[0] == want


@pytest.mark.parametrize("kind", KINDS)
def test_ranges_add_up_to_the_walked_count(wetric_mod, oracle_mod, kind):
    """Wedge ranges are counted by wedge checks, the whole graph by the walk."""
    import torch

    g = far_graph(oracle_mod, kind)
    rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    whole, st = wetric_mod.count(rp, ci, 5, 8192)
    assert st.pair_wedges + st.core_wedges < st.wedges
    cuts = np.sort(np.random.default_rng(5).integers(1, st.wedges, 3))
    cuts = [0, *(int(x) for x in cuts), st.wedges]
    parts = [wetric_mod.count(rp, ci, 5, 8192, wedge_begin=b, wedge_end=e)[0]
             for b, e in zip(cuts, cuts[1:])]
    assert sum(parts) == whole == oracle_mod.count_merge(g)


@pytest.mark.parametrize("k", [1200, 3000])
def test_more_entries_than_room(wetric_mod, oracle_mod, k):
    """A clique below the window, every vertex with one window column: nearly
    every edge makes two entries, more than the room for a quarter above one
    each. The wedge checks take the call -- with 3,000 vertices and host
    columns, after the row chunks have been copied."""
    import torch

    n = 200_000
    at = np.sort(np.random.default_rng(k).choice(n - WINDOW - 10, k, replace=False))
    i, j = np.triu_indices(k, 1)
    g = csr(oracle_mod, n, np.concatenate([at[i], at]),
            np.concatenate([at[j], np.full(k, n - 7)]))
    rest, win, _ = entries(g)
    room = g.m + g.m // 4
    step = 1 << (room.bit_length() - 4)
    assert rest.sum() + win > -(-room // step) * step  # past the room, rounded up
    assert g.m >= 1 << (22 if k == 3000 else 19)
    want = comb3(k) + k * (k - 1) // 2
    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    pinned = (torch.from_numpy(g.row_ptr.view(np.int64)).pin_memory().numpy().view(np.uint64),
              torch.from_numpy(g.col_ind.view(np.int32)).pin_memory().numpy().view(np.uint32))
    for core in (wetric_mod.CORE_OFF, 0, 1000):
        for r, c in ((rp, ci), (rp.int(), ci), (g.row_ptr, g.col_ind), pinned):
            got, st = wetric_mod.count(r, c, 5, 8192, core_len=core)
            assert got == want and st.wedges == st.wedges_counted == oracle_mod.wedge_total(g)


def test_large_sets_go_to_the_wedge_checks(wetric_mod, oracle_mod):
    """More than a tenth of the wedges on rows of several hash sets, from the
    device and in row chunks from the host."""
    import torch

    g = far_graph(oracle_mod, "heavy")
    assert heavy(g, entries(g)[2]) > oracle_mod.wedge_total(g) // 10
    want = oracle_mod.count_merge(g)
    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for core in (wetric_mod.CORE_OFF, 0, 1000, 65_536):
        for r, c in ((rp, ci), (g.row_ptr, g.col_ind)):
            got, st = wetric_mod.count(r, c, 5, 8192, core_len=core)
            assert got == want and st.wedges == st.wedges_counted == oracle_mod.wedge_total(g)


@pytest.mark.parametrize("order", ["id", "random"])
def test_an_order_of_its_own_does_not_slow_the_count(wetric_mod, order):
    """R-MAT scale 18 as drawn and shuffled, oriented by id: the hubs' columns lie
    anywhere. The default count against the wedge checks (it took 3 to 5
    times as long when every rest set was walked)."""
    import torch

    n = 1 << 18
    src, dst = (x.long() for x in wetric_mod.gen_rmat_device(18, 16 << 18, seed=3))
    if order == "random":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(2)
        at = torch.randperm(n, device="cuda", generator=gen)
        src, dst = at[src], at[dst]
    key = torch.unique((torch.minimum(src, dst) * n + torch.maximum(src, dst))[src != dst])
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    ci = (key % n).int()
    torch.cuda.synchronize()

    def ms(**kw):
        runs = [wetric_mod.count(rp, ci, 5, 8192, **kw) for _ in range(6)]
        assert len({c for c, _ in runs}) == 1
        return runs[0][0], sorted(st.exec_ms for _, st in runs)[2]

    (a, default), (b, checks) = ms(), ms(kernel=8)
    assert a == b and default < 1.5 * checks, (default, checks)


def test_batch_far_columns(wetric_mod, oracle_mod):
    """Rows of a batch's own order with more than 48 columns outside their
    graph's window: an even graph of 120,000 vertices, twice, between small
    ones."""
    rng = np.random.default_rng(6)
    n = 120_000
    big = tuple(rng.integers(0, n, 14_400_000).astype(np.uint32) for _ in "sd")
    g = oracle_mod.oriented_from_pairs(*big, n)
    rest, win, _ = entries(g)
    assert rest.sum() > 100_000 and win > 100_000 and rest.sum() + win < g.m + g.m // 4
    want = oracle_mod.count_merge(g)
    tri = tuple(np.array(x, np.uint32) for x in ([0, 1, 2], [1, 2, 0]))
    parts = [tri, big, tri, big]
    src, dst = (np.concatenate([p[q] for p in parts]) for q in (0, 1))
    off = np.concatenate([[0], np.cumsum([p[0].size for p in parts])]).astype(np.uint64)
    b = wetric_mod.Batch(src, dst, off, np.array([3, n, 5, n], np.uint64))
    for _ in range(2):
        assert [int(x) for x in b.count()[0]] == [1, want, 1, want]
    b.free()
    og = wetric_mod.orient_edges(*big, n=n)
    got, st = og.count(5, 8192)
    assert got == want and st.pair_wedges + st.core_wedges < st.wedges


def test_hub_rows_are_shared_out(wetric_mod, oracle_mod):
    """Hubs with up to 60 hash sets among rows of one, few enough that the graph
    is walked: their entries and sets go to several blocks."""
    import torch

    rng = np.random.default_rng(21)
    n, hubs, k = 330_000, 40, 3000
    at = np.sort(rng.choice(n - WINDOW - 70_000, k, replace=False))  # the middle vertices' range
    lengths = rng.choice([900, 1023, 1024, 1025, 2048, 2049, 9000, 33_000, 60_000], hubs)
    src, dst = [], []
    for h, x in zip(rng.choice(at, hubs, replace=False), lengths):
        src.append(np.full(x, h))
        dst.append(h + 1 + rng.choice(n - WINDOW - h - 2, x, replace=False))
    # everybody before a hub points at it and at a few hundred others
    i = np.repeat(at, 300)
    j = rng.choice(at, i.size)
    src += [i, np.repeat(at, hubs)]
    dst += [j, np.tile(np.array([s[0] for s in src[:hubs]]), k)]
    s, d = np.concatenate(src), np.concatenate(dst)
    g = csr(oracle_mod, n, np.minimum(s, d)[s != d], np.maximum(s, d)[s != d])
    rest, win, far = entries(g)
    sets = -(-far[(rest > 0) & (far > PART)] // PART)
    assert sets.max() > 32 and sets.size > 15 and rest[far > PART].max() > 512
    assert g.m >= 1 << 19 and rest.sum() + win < g.m + g.m // 4
    assert heavy(g, far) <= oracle_mod.wedge_total(g) // 10
    want, W = oracle_mod.count_merge(g), oracle_mod.wedge_total(g)
    rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for kw in ({}, {"one_pass": True}, {"core_len": 1000}, {"kernel": 8}):
        got, st = wetric_mod.count(rp, ci, 5, 8192, **kw)
        assert got == want and st.wedges == st.wedges_counted == W, kw
        if "kernel" not in kw:
            assert st.pair_wedges + st.core_wedges < W

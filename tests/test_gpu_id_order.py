"""GPU tests of oriented CSRs whose order is not the one by degree: a row of a
hub that comes early holds most of the vertices, and the columns of its many
short rows are searched for in it (csrc/walk.cuh) instead of merged."""
import numpy as np
import pytest

from conftest import comb3, complete_graph

pytestmark = pytest.mark.gpu
OVER = 2048  # columns from which a row is searched


def id_order(oracle_mod, n, src, dst):
    lo, hi = np.minimum(src, dst).astype(np.int64), np.maximum(src, dst).astype(np.int64)
    key = np.unique((lo * n + hi)[lo != hi])
    rp = np.zeros(n + 1, np.uint64)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return oracle_mod.CSR(rp, (key % n).astype(np.uint32))


def hubs(n, lengths, short, seed):
    """Rows of the given lengths first; the others of 0 to `short` columns, and
    a few of up to 130."""
    rng = np.random.default_rng(seed)
    k = len(lengths)
    src = [np.full(x, i) for i, x in enumerate(lengths)]
    dst = [i + 1 + rng.choice(n - i - 1, x, replace=False) for i, x in enumerate(lengths)]
    d = rng.integers(0, short + 1, n - k)
    d[rng.integers(0, n - k, 30)] = rng.integers(40, 131, 30)
    s = np.repeat(np.arange(k, n), d)
    src.append(s)
    dst.append(np.minimum(s + 1 + rng.integers(0, n, s.size), n - 1))
    return np.concatenate(src), np.concatenate(dst)


@pytest.mark.parametrize("n,lengths,short", [
    (3000, [OVER - 1, OVER, OVER + 1, 2900], 8),  # one launch
    (40_000, [OVER + 1, 5, 30_000], 1),
    (20_000, [OVER, OVER + 1, 15_000, 19_990], 30),  # intersections alone
    (60_000, [40_000, OVER + 1, 50_000], 30),  # with the walk
    (300_000, [250_000, 100_000, OVER - 1, OVER + 40, 200_000], 12),
    (300_000, [50_000], 60)])
def test_long_tails_and_short_rows(wetric_mod, oracle_mod, n, lengths, short):
    import torch

    g = id_order(oracle_mod, n, *hubs(n, lengths, short, n + short))
    want, W = oracle_mod.count_merge(g), oracle_mod.wedge_total(g)
    assert np.diff(g.row_ptr.astype(np.int64)).max() > OVER and want > 0
    rp = torch.from_numpy(g.row_ptr.view(np.int64)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    torch.cuda.synchronize()
    for kw in ({}, {"core_len": wetric_mod.CORE_OFF}, {"core_len": 1000}, {"validate": True},
               {"one_pass": True}, {"kernel": 8}):
        for r in (rp, rp.int()):
            torch.cuda.synchronize()
            got, st = wetric_mod.count(r, ci, 5, 8192, **kw)
            assert got == want and st.wedges == st.wedges_counted == W, kw
    odd = torch.cat([ci[:1], ci])[1:]
    torch.cuda.synchronize()
    assert wetric_mod.count(rp, odd, 5, 8192)[0] == want
    assert wetric_mod.count(g.row_ptr, g.col_ind, 5, 8192)[0] == want


def test_batch_of_long_rows(wetric_mod):
    """Cliques on both sides of the length: rows of a batch's own order."""
    parts = [complete_graph(k) for k in (OVER, OVER + 200, 40, OVER + 2, 3000)]
    off = np.concatenate([[0], np.cumsum([p[0].size for p in parts])]).astype(np.uint64)
    n = [int(p[1].max()) + 1 for p in parts]
    src, dst = (np.concatenate([p[q] for p in parts]) for q in (0, 1))
    for kw in ({}, {"pair_streams": False}):
        b = wetric_mod.Batch(src, dst, off, np.array(n, np.uint64), **kw)
        assert [int(x) for x in b.count()[0]] == [comb3(k) for k in n]
        b.free()


def test_hubs_in_front_do_not_slow_the_count(wetric_mod):
    """A skewed graph in id order: the default count against the wedge checks
    (it took four times as long when every short row was merged)."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    n, pairs = 1 << 18, 6_000_000
    s = (torch.rand(pairs, device="cuda", generator=gen) ** 3 * n).long().clamp_(max=n - 1)
    d = torch.randint(0, n, (pairs,), device="cuda", generator=gen)
    key = torch.unique((torch.minimum(s, d) * n + torch.maximum(s, d))[s != d])
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


def test_a_star_in_front_takes_no_wedge_checks(wetric_mod):
    """Vertex 0 with 400,000 leaves among other edges: 8e10 wedges that close
    nothing, on one row outside the window, and no long row for its tails to
    go to."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    n, leaves = 500_000, 400_000
    s = torch.cat([torch.zeros(leaves, dtype=torch.int64, device="cuda"),
                   torch.randint(1, n, (2_000_000,), device="cuda", generator=gen)])
    d = torch.cat([torch.arange(1, leaves + 1, device="cuda"),
                   torch.randint(1, n, (2_000_000,), device="cuda", generator=gen)])
    key = torch.unique((torch.minimum(s, d) * n + torch.maximum(s, d))[s != d])
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    ci = (key % n).int()
    torch.cuda.synchronize()

    def ms(**kw):
        runs = [wetric_mod.count(rp, ci, 5, 8192, **kw) for _ in range(4)]
        assert len({c for c, _ in runs}) == 1
        return runs[0][0], sorted(st.exec_ms for _, st in runs)[1]

    (a, default), (b, checks) = ms(), ms(kernel=8)
    assert a == b and default < checks / 4, (default, checks)


def test_hubs_with_many_sets_in_front(wetric_mod):
    """300 hubs, then 300,000 vertices with up to 12 columns to them: few wedges
    have both ends on hubs, but each hub has a dozen hash sets (the count took
    2.4 times as long as the wedge checks)."""
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    k, n = 300, 300_300
    i, j = torch.triu_indices(k, k, 1, device="cuda")
    hub = torch.randint(0, k, (12 * (n - k),), device="cuda", generator=gen)
    leaf = torch.arange(k, n, device="cuda").repeat_interleave(12)
    key = torch.unique(torch.cat([i * n + j, hub * n + leaf]))
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    ci = (key % n).int()
    torch.cuda.synchronize()

    def ms(**kw):
        runs = [wetric_mod.count(rp, ci, 5, 8192, **kw) for _ in range(4)]
        assert len({c for c, _ in runs}) == 1
        return runs[0][0], sorted(st.exec_ms for _, st in runs)[1]

    (a, default), (b, checks) = ms(), ms(kernel=8)
    assert a == b and default < 1.5 * checks, (default, checks)

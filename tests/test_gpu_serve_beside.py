"""GPU tests of work beside a resident server's large request: other requests
and the program's own calls run while the resident kernel counts it, not
after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setting(wetric_mod):
    import torch

    rng = np.random.default_rng(1)

    def pairs(n, p):
        return tuple(rng.integers(0, n, p).astype(np.uint32) for _ in "sd")

    mid = pairs(50_000, 400_000)  # past the sort's small tiles
    er = [torch.from_numpy(x.view(np.int32)).cuda() for x in pairs(200_000, 4_000_000)]
    rmat = [torch.from_numpy(x.view(np.int32)).cuda()
            for x in wetric_mod.gen_rmat(18, 16 << 18, seed=4)]
    g = wetric_mod.orient_edges(*rmat, n=1 << 18).download()  # a graph that walks
    rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()
    off = np.array([0, er[0].numel(), er[0].numel() + rmat[0].numel()], np.uint64)
    both = torch.cat([er[0], rmat[0]]), torch.cat([er[1], rmat[1]])
    torch.cuda.synchronize()

    def batch():
        b = wetric_mod.Batch(*both, off, np.array([200_000, 1 << 18], np.uint64))
        counts = [int(x) for x in b.count()[0]]
        b.free()
        return counts

    def orient():
        og = wetric_mod.orient_edges(*er, n=200_000)
        m = og.m
        og.free()
        return m

    big = (*wetric_mod.gen_rmat(23, 16 << 23, seed=2), 1 << 23)
    srv = wetric_mod.Server(resident=True, large_pairs=32 << 20, item_tiles=2048)
    calls = {"request": lambda: srv.wait(srv.submit(*mid, 50_000))[0],
             "count": lambda: wetric_mod.count(rp, ci, 5, 8192)[0],
             "orient": orient, "batch": batch}
    alone = {k: (f(), f())[1] for k, f in calls.items()}  # (the first call loads kernels)
    srv.wait(srv.submit(*big))
    yield srv, big, calls, alone
    srv.close()


@pytest.mark.parametrize("what", ["request", "count", "orient", "batch"])
def test_runs_beside_a_large_request(setting, what):
    import time

    srv, big, calls, alone = setting
    done_first = 0
    for _ in range(5):
        before = srv.stats()["resident_launches"]
        ticket = srv.submit(*big)
        t0 = time.perf_counter()
        while srv.stats()["resident_launches"] == before and time.perf_counter() - t0 < 20:
            time.sleep(0.0005)
        assert calls[what]() == alone[what]
        pending = srv.poll(ticket) is None
        done_first += pending
        if pending:
            srv.wait(ticket)
    assert done_first >= 4, done_first

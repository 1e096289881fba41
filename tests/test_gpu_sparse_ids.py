"""GPU tests of orientation when few of many ids have edges: the long runs of
rows without columns, before, between and behind the others."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHUNK = 65536  # rows that a block fills inside a longer run


@pytest.mark.parametrize("k", [CHUNK // 2, CHUNK - 1, CHUNK, CHUNK + 1, 3 * CHUNK + 5, 2_000_000])
@pytest.mark.parametrize("alone", [0, 1, CHUNK + 7])
def test_runs_of_empty_rows(wetric_mod, k, alone):
    """A matching i -- k + i, then two triangles, behind `alone` ids without
    edges: in the order by degree the ids keep their place, rows
    alone + k ... alone + 2k - 1 are empty."""
    t = alone + 2 * k
    i = np.arange(k)
    src = np.concatenate([alone + i, [t, t, t + 1, t + 3, t + 3, t + 4]]).astype(np.uint32)
    dst = np.concatenate([alone + k + i, [t + 1, t + 2, t + 2, t + 4, t + 5, t + 5]]).astype(np.uint32)
    n = t + 6
    length = np.zeros(n, np.int64)
    length[alone:alone + k] = 1
    length[t:] = [2, 1, 0, 2, 1, 0]
    shuffled = np.random.default_rng(k).permutation(src.size)
    og = wetric_mod.orient_edges(src[shuffled], dst[shuffled], n=n)
    got = og.download()
    og.free()
    assert np.array_equal(got.row_ptr.astype(np.int64), np.concatenate([[0], np.cumsum(length)]))
    assert np.array_equal(got.col_ind, dst)


def test_few_pairs_among_many_ids(wetric_mod):
    """Three pairs among 50,000,000 ids take no longer than three million
    (they took four times as long when three keys had one block)."""
    import torch

    n = 50_000_000
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    many = [torch.randint(0, n, (3_000_000,), device="cuda", generator=gen, dtype=torch.int32)
            for _ in range(2)]
    few = [torch.tensor(x, device="cuda", dtype=torch.int32)
           for x in ([5, 7, n - 1], [7, 9, 5])]
    torch.cuda.synchronize()

    def ms(src, dst):
        t = []
        for _ in range(6):
            start = time.perf_counter()
            og = wetric_mod.orient_edges(src, dst, n=n)
            t.append(time.perf_counter() - start)
            assert og.n == n
            og.free()
        return sorted(t)[2]

    assert ms(*few) < 1.5 * ms(*many)


@pytest.mark.parametrize("dtype", ["int32", "int64"])
def test_no_vertices_launch_nothing(wetric_mod, dtype):
    import torch

    rp = torch.zeros(1, dtype=getattr(torch, dtype), device="cuda")
    ci = torch.zeros(0, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for kw in ({}, {"validate": True}, {"core_len": wetric_mod.CORE_OFF}, {"kernel": 8}):
        count, st = wetric_mod.count(rp, ci, 5, 8192, **kw)
        assert count == 0 and st.wedges == 0 and st.launches == 0, kw

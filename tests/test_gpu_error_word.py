"""GPU tests of the kernels queued behind a scan or a sort: when its look-back
has run out, what it leaves is not complete, so with the error word set they
write nothing. Every array here is complete, so that a kernel that ignored
the word would stay in bounds and be seen by what it wrote; with the word
clear each one does its work."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMEOUT = 7  # kDevLookbackTimeout


def dev(x, dtype):
    import torch

    return torch.from_numpy(np.ascontiguousarray(x, dtype)).cuda()


def call(fn, *args):
    import torch

    torch.cuda.synchronize()
    a = [C.c_void_p(x.data_ptr()) if hasattr(x, "data_ptr") else x for x in args]
    assert fn(*a) == 0
    torch.cuda.synchronize()


@pytest.mark.parametrize("n", [100, 1536, 5000, 300_000])
@pytest.mark.parametrize("bits", [7, 8, 30])
def test_sort(probe, n, bits):
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, n)
    keys = dev(k, np.int64)
    for code in (TIMEOUT, 3, 0):
        a, b, out = (dev(np.full(n, -1), np.int64) for _ in range(3))
        err = dev([code], np.int32)
        call(probe.probe_sort, keys, C.c_uint64(n), C.c_uint32(bits), a, b, out, err)
        assert err.item() == code
        if code:
            assert all((x == -1).all() for x in (a, b, out))
        else:
            assert np.array_equal(out.cpu().numpy(), np.sort(k))


def test_after_a_scan(probe):
    rng = np.random.default_rng(1)
    n = 10_000
    d = rng.integers(0, 6, n)
    rp = np.concatenate([[0], np.cumsum(d)])
    active = d >= 2
    pos = np.concatenate([[0], np.cumsum(active)])
    for code in (TIMEOUT, 0):
        out = dev(np.full(4 * n, -1), np.int64)
        err = dev([code], np.int32)
        call(probe.probe_after_scan, dev(rp, np.int32), C.c_uint64(n), dev(active, np.int32),
             dev(pos, np.int64), out, err)
        got = out.cpu().numpy()
        if code:
            assert (got == -1).all()
        else:
            k = int(active.sum())
            w = (d * (d - 1) // 2)[active]
            assert np.array_equal(got[:k], w) and got[k] == -1
            assert list(got[3 * n:3 * n + 3]) == [pos[n // 2], w[pos[n // 2]], w[pos[n // 2]]]


def test_after_the_walks_sort(probe):
    """Five rows of 60 columns as middle vertices 0, 2, 4, ..., each with one
    entry: a tail of one column, which some of the rows hold."""
    rows, cols = 5, 60
    ci = np.concatenate([np.arange(cols) * 3 + r for r in range(rows)] + [np.arange(rows) * 5 + 9])
    rp = np.arange(rows + 1) * cols
    start_bits, len_bits = 10, 7
    x = np.arange(rows) * 2
    first = rows * cols + np.arange(rows)
    keys = (x << (start_bits + len_bits)) | (first << len_bits) | 1
    want = sum((9 + 5 * r) in ci[r * cols:(r + 1) * cols] for r in range(rows))
    assert 0 < want < rows
    for code in (TIMEOUT, 0):
        start, items = dev(np.full(2 * rows + 1, -1), np.int32), dev(np.full(8 * rows, -1), np.int32)
        counts, out = dev(np.zeros(4), np.int32), dev([0], np.int64)
        err = dev([code], np.int32)
        call(probe.probe_walk, dev(rp, np.int32), dev(rp[1:], np.int32),
             dev(np.arange(rows), np.int32), dev(ci, np.int32), C.c_uint64(ci.size),
             dev(keys, np.int64), C.c_uint32(rows), C.c_uint32(rows), C.c_uint32(start_bits),
             C.c_uint32(len_bits), start, items, counts, out, err)
        if code:
            assert (start == -1).all() and (items == -1).all() and not counts.any()
            assert out.item() == 0
        else:
            assert list(counts.cpu())[:2] == [0, rows] and out.item() == want


def test_after_the_pair_streams_scan(probe):
    rp, ci = dev([0, 2, 3, 3], np.int32), dev([1, 2, 2], np.int32)  # a triangle
    for code, want in ((TIMEOUT, 0), (0, 1)):
        total, err = dev([0], np.int64), dev([code], np.int32)
        call(probe.probe_pairs, rp, ci, dev([0], np.int32), dev([0, 1], np.int64),
             dev([0, 0], np.int32), C.c_uint64(1), total, err)
        assert total.item() == want


def test_after_the_preprocessing_sorts(preprocess_probe):
    rng = np.random.default_rng(2)
    n, N, b = 2000, 30_000, 11
    keys = np.sort(rng.integers(0, n, N) << b | rng.integers(0, n, N))
    uniq = np.unique(keys)
    lo, hi = uniq >> b, uniq & ((1 << b) - 1)
    degrees = np.bincount(lo, minlength=n) + np.bincount(hi, minlength=n)
    for code in (TIMEOUT, 0):
        state, made = dev(np.zeros(N // 4096 + 2), np.int64), dev([-1], np.int64)
        unique, deg = dev(np.full(N, -1), np.int64), dev(np.zeros(n), np.int32)
        rp, ci = dev(np.full(n + 1, -1), np.int64), dev(np.full(N, -1), np.int32)
        err = dev([code], np.int32)
        call(preprocess_probe.probe_after_sort, dev(keys, np.int64), C.c_uint64(N), C.c_uint64(n),
             C.c_uint32(b), state, unique, deg, made, rp, ci, err)
        assert err.item() == code
        if code:
            assert made.item() == -1 and (unique == -1).all() and not deg.any()
            assert (rp == -1).all() and (ci == -1).all()
        else:
            assert made.item() == uniq.size
            assert np.array_equal(unique.cpu().numpy()[:uniq.size], uniq)
            assert np.array_equal(deg.cpu().numpy(), degrees)
            want = np.searchsorted(keys >> b, np.arange(n + 1))
            assert np.array_equal(rp.cpu().numpy(), want)
            assert np.array_equal(ci.cpu().numpy(), keys & ((1 << b) - 1))


def test_after_the_degree_sort(preprocess_probe):
    rng = np.random.default_rng(3)
    n = 3000
    d = rng.integers(0, 9, n)
    rp = np.concatenate([[0], np.cumsum(d)])
    ci = rng.integers(0, n, rp[-1])
    rank = rng.permutation(n)
    row = np.repeat(np.arange(n), d)
    want = np.zeros(n, np.int64)
    want[rank] = np.bincount(row, weights=rank[ci] > rank[row], minlength=n).astype(np.int64)
    for code in (TIMEOUT, 0):
        kept, most, err = dev(np.full(n, -1), np.int32), dev([0], np.int64), dev([code], np.int32)
        call(preprocess_probe.probe_kept, dev(rp, np.int64), dev(ci, np.int32), C.c_uint64(n),
             dev(rank, np.int32), kept, most, err)
        if code:
            assert (kept == -1).all() and most.item() == 0
        else:
            assert np.array_equal(kept.cpu().numpy(), want) and most.item() == want.max()

"""The words that look-back scans publish between their tiles
(csrc/primitives.cuh): wedge prefixes are 64 bits wide."""
import ctypes as C

import numpy as np
import pytest

AGG, INCL, POISON = 1, 2, 3
VALUES = [0, 1, (1 << 48) - 1, 1 << 48, 1 << 49, (1 << 49) + 5, (1 << 50) - 1, 1 << 62,
          (1 << 64) - 1]


def words(probe, flag, value):
    w = (C.c_uint64 * 2)()
    probe.probe_tile_words(flag, C.c_uint64(value), w)
    return list(w)


def read(probe, w):
    v = C.c_uint64()
    return probe.probe_tile_read((C.c_uint64 * 2)(*w), C.byref(v)), v.value


@pytest.mark.parametrize("value", VALUES)
def test_tile_words_hold_64_bits(probe, value):
    for flag in (AGG, INCL):
        assert read(probe, words(probe, flag, value)) == (flag, value)
    assert read(probe, words(probe, POISON, value))[0] == POISON


def test_tile_words_of_two_values_are_not_ready(probe):
    for a in VALUES:
        for b in VALUES:
            agg, incl = words(probe, AGG, a), words(probe, INCL, b)
            assert read(probe, [agg[0], incl[1]])[0] == 0
            assert read(probe, [incl[0], agg[1]])[0] == 0
            assert read(probe, [0, agg[1]])[0] == 0 and read(probe, [agg[0], 0])[0] == 0
            bad = words(probe, POISON, 0)
            assert read(probe, [bad[0], agg[1]])[0] == POISON
            assert read(probe, [agg[0], bad[1]])[0] == POISON


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 4096, 4097, 128 * 4096, 129 * 4096 + 1, 700_001])
def test_scan_of_large_values(probe, wetric_mod, n):
    """Few large values among small ones: single values, tile totals and
    prefixes on both sides of 2^48 and up to 2^64."""
    import torch

    rng = np.random.default_rng(n)
    for big in (1 << 47, 1 << 49, (1 << 59) - 3):
        x = rng.integers(0, 1000, n).astype(np.uint64)
        k = max(1, min(n, ((1 << 64) - 1) // big // 2, n // 50))
        x[rng.choice(n, k, replace=False)] = big
        x[0] = big
        d = torch.from_numpy(x.view(np.int64)).cuda()
        out = torch.empty(n + 1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        err = C.c_uint32()
        assert probe.probe_scan_u64(C.c_void_p(d.data_ptr()), C.c_uint64(n),
                                    C.c_void_p(out.data_ptr()), C.byref(err)) == 0
        assert err.value == 0
        want = np.concatenate([np.zeros(1, np.uint64), np.cumsum(x, dtype=np.uint64)])
        assert np.array_equal(out.cpu().numpy().view(np.uint64), want)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["int32", "int64"])
def test_wedge_total_past_48_bits(wetric_mod, dtype):
    """Rows in id order with a hub of 2^25 columns and more (2^49 wedges), in
    the first tile of the prefix and in later ones."""
    import torch

    n = 50_000
    d = np.full(n, 7, np.int64)
    hubs = [0, 1, 4096, 30_000] if dtype == "int32" else list(range(0, n, 2500))
    d[hubs] = (1 << 25) + 9 if dtype == "int32" else (1 << 29) - 1
    rp = torch.zeros(n + 1, dtype=torch.int64)
    rp[1:] = torch.cumsum(torch.from_numpy(d), 0)
    W = sum(int(x) * (int(x) - 1) // 2 for x in d)
    assert (1 << 50) < W < (1 << 64)
    got, longest = wetric_mod.wedge_total(rp.to(getattr(torch, dtype)).cuda())
    assert got == W and longest == d.max()

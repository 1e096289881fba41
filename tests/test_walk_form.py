"""Which way a graph is counted below its core (csrc/walk.cuh): by row
intersections alone, with the column walk, or by the wedge checks when the
walk's 64-bit entries have no room for the graph's row numbers, column
indices and tail lengths."""
import ctypes as C

import numpy as np
import pytest

MERGE, WALK, WEDGES = 0, 1, 2


def form(probe, n, m, edges, long_rows, longest, long_wedges):
    return probe.probe_walk_form(*(C.c_uint64(x) for x in
                                   (n, m, edges, long_rows, longest, long_wedges)))


def test_large_graphs_with_hubs_are_not_merged(probe):
    """Whatever the size, a graph whose long rows want the walk never has them
    intersected edge by edge."""
    for m_bits in range(20, 31):
        m = (1 << m_bits) + 12_345
        for rows in (1, 1000, m // 200, m // 49):
            for longest in (129, 1000, 5000, 100_000, 1 << 22):
                if rows * 49 + longest > m:
                    continue
                got = form(probe, m // 8, m, m, rows, longest, 1 << 40)
                room = 1 + max(1, (rows - 1).bit_length()) + m.bit_length() + longest.bit_length()
                assert got == (WALK if room <= 64 else WEDGES), (m, rows, longest)


def test_forms_at_known_sizes(probe):
    # R-MAT, edge factor 16: (n, m, long rows, longest row) of scales 22, 24
    assert form(probe, 1 << 22, 64_153_649, 64_000_000, 300_000, 1100, 1 << 33) == WALK
    assert form(probe, 1 << 24, 260_000_000, 260_000_000, 1_200_000, 2000, 1 << 36) == WALK
    # past 64 bits
    assert form(probe, 1 << 27, (1 << 31) - 1, (1 << 31) - 1, 10_000_000, 8000, 1 << 38) == WEDGES
    # no long rows, few edges, or short long rows: intersections
    assert form(probe, 1 << 27, (1 << 31) - 1, (1 << 31) - 1, 0, 48, 0) == MERGE
    assert form(probe, 1 << 27, 1 << 30, (1 << 19) - 1, 1 << 22, 1 << 20, 1 << 40) == MERGE
    assert form(probe, 1 << 27, (1 << 31) - 1, (1 << 31) - 1, 1 << 23, 128, 1 << 24) == MERGE


def band(n, d, hub):
    """Row v holds v + 1 ... v + d (to n - 1), row 0 the first `hub` instead."""
    import torch

    length = torch.clamp(n - 1 - torch.arange(n, device="cuda"), max=d)
    length[0] = hub
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(length, 0)
    m = int(rp[-1])
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), length)
    ci = row + 1 + torch.arange(m, device="cuda") - rp[row]
    return rp, ci.int(), length.cpu().numpy()


@pytest.mark.gpu
def test_entries_past_64_bits(probe, wetric_mod):
    """2.1 million rows of 49 columns and one of 16,500: one bit too many."""
    n, d, hub = 2_100_100, 49, 16_500
    rp, ci, length = band(n, d, hub)
    m, long = ci.numel(), length > 48
    w = length.astype(object) * (length - 1) // 2
    assert form(probe, n, m, m, int(long.sum()), hub, int(w[long].sum())) == WEDGES

    def in_band(k):  # pairs of k consecutive ids at most d apart
        return d * k - d * (d + 1) // 2

    # three ids at most d apart without row 0, and row 0's closing pairs
    want = (n - 1) * d * (d - 1) // 2 - sum(d * (d - 1) // 2 - j * (j - 1) // 2
                                            for j in range(d)) + in_band(hub)
    for kw in ({}, {"core_len": wetric_mod.CORE_OFF}, {"kernel": 8}):
        got, st = wetric_mod.count(rp.int(), ci, 5, 8192, **kw)
        assert got == want, kw
        assert st.wedges == int(w.sum())

"""The host threads that copy staged pieces (csrc/stage_workers.h): whole
copies at the edges of their blocks, from one caller, from as many as have
slots, and from more; with gaps in which the threads go to sleep."""
import ctypes as C

import pytest

MB = 1 << 20


@pytest.mark.parametrize("callers", [1, 2, 4])
@pytest.mark.parametrize("gap_ms", [0, 6])
def test_copies_are_whole(probe, callers, gap_ms):
    sizes = [0, 1, MB - 1, MB, MB + 1, 3 * MB + 7, 16 * MB] if gap_ms else \
        [5, MB - 1, MB, 2 * MB + 3, 9 * MB + 1] * 4
    a = (C.c_uint64 * len(sizes))(*sizes)
    assert probe.probe_stage_copies(a, len(sizes), callers, 3, gap_ms) == 0

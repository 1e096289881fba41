"""GPU tests of inputs that only the kernels' own checks keep in bounds, and of
results at the widths where packed words end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n,m", [(1_000_000, 200_000), (300_001, 131_072), (400_000, 4_300_000)])
def test_overlapping_rows_are_rejected(wetric_mod, dtype, n, m):
    """Offsets 0, m, 0, m, ..., m: half of the rows hold every column, so there
    are many more long rows than m columns have room for, while every offset
    is at most m and the first and last are right."""
    import torch

    rp = np.zeros(n + 1, dtype)
    rp[1::2] = m
    rp[n] = m
    length = np.diff(rp.astype(np.int64))
    assert (length > 48).sum() > m // 49 + 1  # past the room
    assert (length < 0).any() and rp[0] == 0 and rp[n] == m and rp.max() == m
    ci = np.arange(m, dtype=np.int32) % n
    for r, c in ((torch.from_numpy(rp).cuda(), torch.from_numpy(ci).cuda()),
                 (rp.view(np.uint32 if dtype == np.int32 else np.uint64), ci.view(np.uint32))):
        for core in (0, wetric_mod.CORE_OFF):
            with pytest.raises(wetric_mod.WetricError) as e:
                wetric_mod.count(r, c, 5, 8192, core_len=core)
            assert e.value.status == 1, e.value
    # the device still counts
    assert wetric_mod.count(np.array([0, 2, 3, 3], np.uint64), np.array([1, 2, 2], np.uint32))[0] == 1


@pytest.mark.parametrize("most", [0, 1, 1 << 27, (1 << 32) - 1, 1 << 40])
def test_a_warps_hits_are_summed_in_64_bits(probe, wetric_mod, most):
    import ctypes as C

    import torch

    hits = np.random.default_rng(1).integers(0, most + 1, 32)
    hits[0] = most
    d = torch.from_numpy(hits).cuda()
    total = torch.full((1,), 5, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    assert probe.probe_add_hits(C.c_void_p(d.data_ptr()), C.c_void_p(total.data_ptr())) == 0
    assert total.item() == 5 + int(hits.sum())

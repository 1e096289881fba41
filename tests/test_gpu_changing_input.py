"""GPU test of pairs that another stream changes while they are oriented, as a
program does that forgets to order its own writes before the call: the graph
is then one of many, but it is a whole one, and nothing outside the call's
buffers is touched."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pairs,n", [(3_000_000, 1 << 16), (40_000, 1 << 10), (12_000_000, 1 << 20)])
def test_orienting_pairs_that_change(wetric_mod, pairs, n):
    import torch

    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    kinds = [torch.randint(0, n, (pairs,), device="cuda", generator=gen, dtype=torch.int32),
             torch.randint(0, 7, (pairs,), device="cuda", generator=gen, dtype=torch.int32),
             torch.full((pairs,), n - 1, device="cuda", dtype=torch.int32)]
    src, dst = kinds[0].clone(), kinds[0].roll(1)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for i in range(12):
        with torch.cuda.stream(side):
            for j in range(30):
                (src if j & 1 else dst).copy_(kinds[(i + j) % 3])
        og = wetric_mod.orient_edges(src, dst, n=n)
        g = og.download()
        side.synchronize()
        rp, ci = g.row_ptr.astype(np.int64), g.col_ind.astype(np.int64)
        assert rp[0] == 0 and rp[-1] == ci.size <= pairs and (np.diff(rp) >= 0).all()
        row = np.repeat(np.arange(n), np.diff(rp))
        assert (ci > row).all() and (ci < n).all()
        assert ((np.diff(ci) > 0) | (np.diff(row) > 0)).all()  # sorted, no repeats
        og.free()

"""GPU test of counts whose blocks end early so that other streams get SMs
(one_pass): the column walk hands out its items in advance there, a few to a
block."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edge_factor", [16, 64])
def test_one_pass_costs_little(wetric_mod, edge_factor):
    """16 items to a block took half as long again as the default launch."""
    import torch

    src, dst = wetric_mod.gen_rmat(18, edge_factor << 18, seed=4)
    og = wetric_mod.orient_edges(src, dst, n=1 << 18)

    def ms(**kw):
        runs = [og.count(5, 8192, **kw) for _ in range(8)]
        assert len({c for c, _ in runs}) == 1
        return runs[0][0], sorted(st.exec_ms for _, st in runs)[3]

    torch.cuda.synchronize()
    (a, default), (b, short) = ms(), ms(one_pass=True)
    og.free()
    assert a == b and short < 1.25 * default, (short, default)

"""GPU tests under limited device memory: what the wedge checks have room for,
the default count has room for too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core", [0, 20_000])
def test_default_count_fits_where_the_wedge_checks_fit(wetric_mod, oracle_mod, core):
    """From no budget up past the default count's whole need: each budget either
    gives the count or, where the wedge checks do not fit either, ENOMEM."""
    import torch

    src, dst = wetric_mod.gen_rmat(18, 16 << 18, seed=9)
    g = oracle_mod.oriented_from_pairs(src, dst)
    want = oracle_mod.count_merge(g)
    rp = torch.from_numpy(g.row_ptr.astype(np.int32)).cuda()
    ci = torch.from_numpy(g.col_ind.view(np.int32)).cuda()

    def fits(budget, **kw):
        try:
            wetric_mod.set_hbm_budget(budget)
            assert wetric_mod.count(rp, ci, 5, 8192, core_len=core, **kw)[0] == want
            return True
        except wetric_mod.WetricError as e:
            assert e.status == wetric_mod.ENOMEM, e
            return False
        finally:
            wetric_mod.set_hbm_budget(0)

    budgets = [int((1 << 20) * 1.04 ** i) for i in range(140)]  # 1 MB to 240 MB
    checks = [fits(b, kernel=8) for b in budgets]
    default = [fits(b) for b in budgets]
    assert checks.count(False) > 3 and checks[-1]
    assert [b for b, c, d in zip(budgets, checks, default) if c and not d] == []

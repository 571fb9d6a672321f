"""K at thresholds of zero and below ("keep everything"): pairs whose FP32 bound underflows
to 0 stay in a list built with a negative threshold, their quartets pass the screens, and
the quartets beside them in a warp must not be lost."""
import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("thre,thresp", [(-1.0, 0.0), (-1.0, -1.0), (0.0, 0.0), (-1.0, 1e-12)])
@pytest.mark.parametrize("symm", [True, False])
def test_zero_bounds_lose_no_quartets(ls, thre, thresp, symm):
    if not port.available():
        pytest.skip("oracle port not built")
    from lightspeed_b200.geometry import water_cluster
    bas = ls.Basis.from_gbs_file(water_cluster(2, seed=3), "6-31gs")
    rng = np.random.default_rng(11)
    X = rng.standard_normal((bas.nao, 5)) * 0.3
    D = X @ X.T if symm else X @ rng.standard_normal((5, bas.nao)) * 0.3
    pb = port.Basis(bas.primitives)
    pp = port.Pairs(pb, pb, True, thre)
    assert np.any(pp.bound == 0.0) == (thre < 0.0)   # the tight s pairs of the two oxygens
    _, nk = port.count_quartets(pp, pp, D, D, symm, thresp)
    Kp = port.exchange(pp, pp, D, symm, thresp)
    pl = ls.PairList.build_schwarz(bas, bas, True, thre)
    res, ew = ls.ResourceList.build(), ls.Ewald.coulomb()
    scale = max(1.0, np.max(np.abs(Kp)))
    try:
        for merge in (False, True):
            ls.set_merge(merge)
            ls.set_precision(ls.PREC_FP64)
            ls.reset_stats()
            K = ls.IntBox.exchange(res, ew, pl, pl, ls.Tensor.array(D), symm, thresp, thresp).np.copy()
            if not merge:
                assert ls.stats()["k_quartets"] == nk
            # the same quartets, FP64 sums in another order (the merged build's extra ones are
            # below thresp each)
            assert np.max(np.abs(K - Kp)) < 1e-12 * scale + 4.0 * nk / bas.nao ** 2 * max(0.0, thresp)
            ls.set_precision(ls.PREC_MIXED)
            ls.reset_stats()
            Km = ls.IntBox.exchange(res, ew, pl, pl, ls.Tensor.array(D), symm, thresp, 1e-5).np
            assert ls.stats()["quartets_fp32"] > 0
            # FP32 quartets are below 1e-5 each
            assert np.max(np.abs(Km - K)) < 1e-6
    finally:
        ls.set_merge(False)
        ls.set_precision(ls.PREC_MIXED)

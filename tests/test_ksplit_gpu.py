"""K classes with few (prim2, prim4) tasks cut the partner-1 rows into stripes that
may start inside a shell segment: the quartet set must stay the reference's, and K
that of the CPU restatement, where the screens bite inside rows and segments."""
import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("system,basis,thre,symm", [
    ("w1", "6-31gs", 1e-14, True), ("w1", "6-31gs", 1e-6, False), ("w2", "cc-pvdz", 1e-9, True),
    ("w3", "6-31gs", 1e-10, False), ("c2", "cc-pvdz", 1e-11, True), ("w1", "sto-3g", 1e-12, True)])
def test_split_rows_quartets_and_values(ls, system, basis, thre, symm):
    if not port.available():
        pytest.skip("oracle port not built")
    from lightspeed_b200.geometry import alkane, water_cluster
    n = int(system[1:])
    mol = water_cluster(n, seed=4) if system[0] == "w" else alkane(n)
    bas = ls.Basis.from_gbs_file(mol, basis)
    rng = np.random.default_rng(7)
    X = rng.standard_normal((bas.nao, 5)) * 0.3
    D = X @ X.T if symm else X @ rng.standard_normal((5, bas.nao)) * 0.3
    pl = ls.PairList.build_schwarz(bas, bas, True, thre)
    pb = port.Basis(bas.primitives)
    pp = port.Pairs(pb, pb, True, thre)
    _, nk = port.count_quartets(pp, pp, D, D, symm, thre)
    Kp = port.exchange(pp, pp, D, symm, thre)
    res, ew = ls.ResourceList.build(), ls.Ewald.coulomb()
    try:
        for merge in (False, True):
            ls.set_merge(merge)
            ls.set_precision(ls.PREC_FP64)
            ls.reset_stats()
            K = ls.IntBox.exchange(res, ew, pl, pl, ls.Tensor.array(D), symm, thre, thre).np.copy()
            if not merge:
                assert ls.stats()["k_quartets"] == nk
                # the same quartets, FP64 sums in another order
                assert np.max(np.abs(K - Kp)) < 1e-12 * max(1.0, np.max(np.abs(Kp)))
            else:
                # a superset: the extra terms are below thre, and an element has nk / nao^2 quartets on average
                assert np.max(np.abs(K - Kp)) < 4.0 * nk / bas.nao ** 2 * thre + 1e-12
            ls.set_precision(ls.PREC_MIXED)
            Km = ls.IntBox.exchange(res, ew, pl, pl, ls.Tensor.array(D), symm, thre, max(1e-5, 10 * thre)).np
            # FP32 quartets are below thredp each; their rounding is 6e-8 of that, over at most nk of them per element
            assert np.max(np.abs(Km - K)) < 1e-6
    finally:
        ls.set_merge(False)
        ls.set_precision(ls.PREC_MIXED)

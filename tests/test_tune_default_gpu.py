"""The autotuner has the default J schedule among its candidates: on a molecule so small that
every fixed ket chunk leaves most of the GPU idle, it keeps the default (table entry 0)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_small_molecule_keeps_the_default_chunks(ls):
    from lightspeed_b200.geometry import water_cluster
    bas = ls.Basis.from_gbs_file(water_cluster(4, seed=8), "6-31gs")
    pl = ls.PairList.build_schwarz(bas, bas, True, 1e-14)
    X = np.random.default_rng(1).standard_normal((bas.nao, 8)) / np.sqrt(bas.nao)
    D, res, ew = ls.Tensor.array(X @ X.T), ls.ResourceList.build(), ls.Ewald.coulomb()
    nherm = 7   # Hermite classes up to (f|f): the table's first nherm^2 entries are J's
    sizes = np.zeros(nherm, int)
    for p in pl.pairlists:
        sizes[p.L1 + p.L2] += len(p.pairs)
    saved = ls.get_tune_table()
    ls.set_precision(ls.PREC_FP64)
    try:
        J0 = ls.IntBox.coulomb(res, ew, pl, pl, D, 1e-14, 1e-14).np.copy()
        ls.set_autotune(True)
        ls.IntBox.coulomb(res, ew, pl, pl, D, 1e-14, 1e-14)
        ls.set_autotune(False)
        table = np.array(ls.get_tune_table()[:nherm * nherm]).reshape(nherm, nherm)
        # classes with several fixed chunks' worth of kets, walked serially by a few CTAs each
        served = np.outer(sizes > 0, sizes > 256)
        assert served.sum() >= 10
        assert np.count_nonzero(table[served] == 0) > 0.8 * served.sum()
        J1 = ls.IntBox.coulomb(res, ew, pl, pl, D, 1e-14, 1e-14).np
        assert np.max(np.abs(J1 - J0)) < 1e-10
    finally:
        ls.set_autotune(False)
        ls.set_tune_table(saved)
        ls.set_precision(ls.PREC_MIXED)

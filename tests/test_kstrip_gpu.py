"""Mixed-precision K between different bases: the FP32 pass adds into a K in strip layout,
which the build joins with the FP64 pass's by the shells of basis 1. Rectangular K13, one
density and more, a merged list on one side of a plain one."""
import numpy as np
import pytest

from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("names", [("cc-pvdz", "6-31gs", "6-31gs", "6-31gs"), ("6-31gs", "6-31gs", "cc-pvdz", "6-31gs"),
                                   ("cc-pvdz", "6-31gs", "sto-3g", "cc-pvdz"), ("6-31gs", "cc-pvdz", "cc-pvdz", "sto-3g")])
@pytest.mark.parametrize("ndens", [1, 5])
def test_mixed_k_of_different_bases(ls, names, ndens):
    if not port.available():
        pytest.skip("oracle port not built")
    from lightspeed_b200.geometry import water_cluster
    mol = water_cluster(3, seed=9)
    bas = [ls.Basis.from_gbs_file(mol, b) for b in names]
    thre, thredp = 1e-12, 1e-5
    pl = [ls.PairList.build_schwarz(bas[k], bas[k + 1], False, thre) for k in (0, 2)]
    rng = np.random.default_rng(21)
    Ds = [rng.standard_normal((bas[1].nao, 4)) @ rng.standard_normal((4, bas[3].nao)) * 0.1 for _ in range(ndens)]
    pb = [port.Basis(b.primitives) for b in bas]
    pp = [port.Pairs(pb[k], pb[k + 1], False, thre) for k in (0, 2)]
    Kp = [port.exchange(pp[0], pp[1], D, False, thre) for D in Ds]
    assert Kp[0].shape == (bas[0].nao, bas[2].nao) and bas[0].nao != bas[2].nao
    _, nk = port.count_quartets(pp[0], pp[1], np.ones((bas[2].nao, bas[3].nao)), Ds[0], False, thre)
    res, ew = ls.ResourceList.build(), ls.Ewald.coulomb()
    run = lambda dp: [K.np.copy() for K in ls.IntBox.exchangeMulti(
        res, ew, pl[0], pl[1], [ls.Tensor.array(D) for D in Ds], False, thre, dp)]
    try:
        for merge in (False, True):
            ls.set_merge(merge)
            ls.set_precision(ls.PREC_FP64)
            K64 = run(thre)
            ls.set_precision(ls.PREC_MIXED)
            ls.reset_stats()
            Km = run(thredp)
            s = ls.stats()
            assert s["quartets_fp32"] > 0 and s["quartets_fp64"] > 0
            for p, a, b in zip(Kp, K64, Km):
                # several densities (and merged copies) screen together: a superset of one's
                # quartets, the extra ones below thre each
                assert np.max(np.abs(a - p)) < 1e-12 * max(1.0, np.max(np.abs(p))) + 4.0 * nk / p.size * thre
                # FP32 quartets are below thredp each, their rounding 6e-8 of that
                assert np.max(np.abs(b - a)) < 1e-6
    finally:
        ls.set_merge(False)
        ls.set_precision(ls.PREC_MIXED)
